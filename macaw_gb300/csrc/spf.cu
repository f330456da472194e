// SPF derivatives of the grid modes (derivatives.f90:94-153) for sm_103a: digit
// products on the tensor cores (fixed.cuh) for the operator sum and the contractions,
// FP64 for the small solve:
//  (1) dphi = f sum_k ophi_k rhom1MF_k^T, 64 grid rows per CTA;
//  (2) the contractions phi^H phi and phi^H dphi;
//  (3) solve (phi^H phi) X = phi^H dphi (zposv 'U'), dphi -= phi X.
// Up to eight SPFs a CTA contracts its own rows after (1), from shared memory; modes of
// at most 64 grid points then go through (3) in the same CTA, one launch in all, larger
// ones through a second launch that adds the CTAs' contractions.  More SPFs: (2) is the
// contraction kernel (fixed.cu), three launches.
#include "kernels.cuh"
#include "fixed.cuh"

#define SPF_THREADS 256
#define SPF_CHUNK 9      // steps of eight columns between flushes: 5 x 16 x 8 x 2^14 < 2^24 per half
#define SPF_COLS (8 * SPF_CHUNK)

#define SPF_PITCH (SPF_ROWS + 2)   // staged rows of a column: the lanes' 16-byte reads meet no bank twice

// Shared operands of row_products.
struct RowShared {
  cplx x[SPF_CHUNK][8][SPF_PITCH];         // the CTA's rows of a chunk of steps
  union {
    uint2 W[SPF_CHUNK][2][FX_NS][32];     // digits of eight columns of the matrix (j2 = q and q + 4)
    struct {
      unsigned char small[sizeof(uint2) * SPF_CHUNK * 2 * FX_NS * 32 - 8192 - 2048];
      float tother[4][2][2][32];           // the second warps' sums of |x||rm| and their
      cplx other[4][2][2][32];             // sums, once W is read
    };
  };
  unsigned colmag[8], top;                 // largest elements of the columns j1 (scaled), of the matrix
  unsigned scale[SPF_COLS];                // the columns' scaling
};
// the scaling of a column whose rm are zero: its x, brought out of range by it, count for
// nothing, and the digits of either are zero
#define SPF_EMPTY 0x7ff00000u
#define SPF_SCALE_MAX 400

__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Rows row0 .. row0 + 63 of the columns 8 s0 .. 8 (s0 + ns) - 1 on their way into S.x
// (zeros beyond G and ncols); copy_async_wait and a barrier complete it.
template <typename Col>
__device__ __forceinline__ void stage_rows(RowShared& S, int s0, int ns, Col&& col, int ncols, int G, int row0) {
  const int row = threadIdx.x & (SPF_ROWS - 1);
#pragma unroll 2
  for (int j = threadIdx.x / SPF_ROWS; j < 8 * ns; j += SPF_THREADS / SPF_ROWS) {
    cplx* to = &S.x[j >> 3][j & 7][row];
    if (row0 + row < G && 8 * s0 + j < ncols) copy_async16(to, col(8 * s0 + j).x + row0 + row);
    else *to = mkc(0.0, 0.0);
  }
}

// 2^e as FP32 for e <= 0, zero where that is no normal number
__device__ __forceinline__ float spf_pow2(int e) { return e > -127 ? __int_as_float((e + 127) << 23) : 0.f; }

// The CTA's rows row0 .. row0 + 63 of sum_j x(row, j) rm(j1, j) over ncols columns for all
// j1 < n: warps w and w + 4 own 16 rows (the MMA's rows) and every second step, the
// columns are the (re, im) of four j1.  Column j of x is multiplied and rm(., j) divided
// by a power of two that makes the rm(., j) alike in size, whatever the operators' units;
// then a row has one exponent per chunk of steps, a column j1 of the matrices another.
// col(j) returns the j-th column of x and of rm, a step is eight of them (whatever
// operators they belong to); the first chunk is staged already.
// put(row, j1, value) takes the results (warps 0 - 3); rows from G on are skipped.  The
// matrices are cut while the rows are on their way.  Operands outside the exponent range
// are multiplied in FP64, and so are elements whose sum of |x||rm| (one more MMA, on the
// leading digits) is below 2^-6 .. 2^-8 of the product of the largest elements.
template <typename Col, typename Put>
__device__ __forceinline__ void row_products(RowShared& S, int ncols, Col&& col, int n, int G, int row0, Put&& put) {
  constexpr int NS = FX_NS;
  const int nsteps = (ncols + 7) / 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int half = warp >> 2, lr = 16 * (warp & 3) + g;   // the lane's rows: lr, lr + 8
  auto& other = S.other;
  for (int j0 = 0; j0 < n; j0 += 8) {   // eight outputs per pass
    cplx sum[2][2];                     // [group of four j1][row]
    // sums of |x||rm|, and of the products of largest elements, both times 2^-eref
    float tsum[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, bsum[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    int eref[2][2] = {{0, 0}, {0, 0}};
    for (int s0 = 0; s0 < nsteps; s0 += SPF_CHUNK) {
      const int ns = min(SPF_CHUNK, nsteps - s0);
      if (s0 || (j0 && nsteps > SPF_CHUNK)) {
        __syncthreads();   // the previous chunk is read
        stage_rows(S, s0, ns, col, ncols, G, row0);
      }
      if (tid < 8) S.colmag[tid] = 0u;
      if (tid == 8) S.top = 0u;
      __syncthreads();
      const int nc = min(8, n - j0);
      // (j, j1): at most three per thread, the eight of a column in neighbouring lanes
      constexpr int PER = (64 * SPF_CHUNK + SPF_THREADS - 1) / SPF_THREADS;
      unsigned m[PER], rmag[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int e = tid + i * SPF_THREADS, j = 8 * s0 + (e >> 3);
        m[i] = e < 64 * ns && j < ncols && (e & 7) < nc ? fx_mag(col(j).rm[j0 + (e & 7)]) : 0u;
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        rmag[i] = m[i];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) rmag[i] = max(rmag[i], __shfl_xor_sync(0xffffffffu, rmag[i], o));
        if ((tid & 7) == 0 && rmag[i]) atomicMax(&S.top, rmag[i]);
      }
      __syncthreads();
      const unsigned top = S.top & FX_EBITS;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int e = tid + i * SPF_THREADS;
        if (e >= 64 * ns) break;
        const unsigned b = min(top - (rmag[i] & FX_EBITS), (unsigned)SPF_SCALE_MAX << 20);
        if ((e & 7) == 0) S.scale[e >> 3] = rmag[i] ? b : SPF_EMPTY;
        if (m[i]) atomicMax(&S.colmag[e & 7], m[i] + b);
      }
      __syncthreads();
      bool bad = tid < nc && !fx_ok(S.colmag[tid]);
      for (int w = warp; w < 2 * ns; w += SPF_THREADS / 32) {
        const int t = w & 1, s = w >> 1, j1 = 4 * t + (g >> 1);
        if (4 * t >= nc) continue;
        const int jl = 8 * s + q, jc = 8 * s0 + jl;
        unsigned d0[NS], d1[NS];
        const cplx m0 = (j1 < nc && jc < ncols) ? col(jc).rm[j0 + j1] : mkc(0, 0);
        const cplx m1 = (j1 < nc && jc + 4 < ncols) ? col(jc + 4).rm[j0 + j1] : mkc(0, 0);
        const unsigned em = fx_ebits(S.colmag[j1]), b0 = S.scale[jl], b1 = S.scale[jl + 4];
        fx_digits(m0.x, m0.y, em - b0, em - b0, d0);
        fx_digits(m1.x, m1.y, em - b1, em - b1, d1);
#pragma unroll
        for (int i = 0; i < NS; ++i) {   // column re: (Mr, -Mi); column im: (Mi, Mr)
          const unsigned w0 = (g & 1) ? __byte_perm(d0[i], d0[i], 0x1032) : d0[i] ^ 0x80000000u;
          const unsigned w1 = (g & 1) ? __byte_perm(d1[i], d1[i], 0x1032) : d1[i] ^ 0x80000000u;
          S.W[s][t][i][lane] = make_uint2(w0, w1);
        }
      }
      copy_async_wait();
      __syncthreads();
      unsigned mag[2];
      {
        int most[2] = {0, 0};        // scaled
        unsigned raw[2] = {0u, 0u};
#pragma unroll 3
        for (int s = 0; s < ns; ++s)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const unsigned b = S.scale[8 * s + q + 4 * h];
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              const unsigned x = fx_mag(S.x[s][q + 4 * h][lr + 8 * f]);
              raw[f] = max(raw[f], b == SPF_EMPTY && x < FX_EBITS ? 0u : x);
              most[f] = max(most[f], (int)(x - b));
            }
          }
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          most[f] = max(most[f], __shfl_xor_sync(0xffffffffu, most[f], 1));
          most[f] = max(most[f], __shfl_xor_sync(0xffffffffu, most[f], 2));
          mag[f] = (unsigned)most[f];
          bad = bad || !fx_ok(mag[f]) || raw[f] >= FX_EBITS || (raw[f] && !mag[f]);
        }
      }
      const unsigned eb[2] = {fx_ebits(mag[0]), fx_ebits(mag[1])};
      if (__syncthreads_or(bad)) {   // the pass in FP64
        for (int e = tid; e < SPF_ROWS * nc; e += SPF_THREADS) {
          const int row = row0 + (e & (SPF_ROWS - 1)), j1 = j0 + e / SPF_ROWS;
          if (row >= G) continue;
          cplx acc = mkc(0, 0);
          for (int j = 0; j < ncols; ++j) cfma(acc, col(j).x[row], col(j).rm[j1]);
          put(row, j1, acc);
        }
        goto next_pass;
      }
      {
        float c[2][NS][4], ct[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            ct[t][k] = 0.f;
#pragma unroll
            for (int i = 0; i < NS; ++i) c[t][i][k] = 0.f;
          }
        for (int s = half; s < ns; s += 2) {
          unsigned A[NS][4], ta[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const unsigned b = S.scale[8 * s + q + 4 * h];
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              unsigned d[NS];
              const cplx x = S.x[s][q + 4 * h][lr + 8 * f];
              fx_digits(x.x, x.y, eb[f] + b, eb[f] + b, d);
#pragma unroll
              for (int i = 0; i < NS; ++i) A[i][2 * h + f] = d[i];
              ta[2 * h + f] = fx_lead(d[0], d[1]);
            }
          }
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (4 * t < nc) {
              uint2 w0;
#pragma unroll
              for (int i = 0; i < NS; ++i) {
                const uint2 w = S.W[s][t][i][lane];
                if (i == 0) w0 = w;
                if (i == 1) fx_mma16(ct[t], ta, fx_lead(w0.x, w.x), fx_lead(w0.y, w.y), false);
#pragma unroll
                for (int j = 0; j + i < NS; ++j) fx_mma16(c[t][i + j], A[j], w.x, w.y, false);
              }
            }
          }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (4 * t < nc) {
            const unsigned cm = S.colmag[4 * t + q], em = fx_ebits(cm);
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              const unsigned es = fx_exp(em, eb[f], 44);
              const cplx v = mkc(fx_double(fx_join_wide(c[t], 2 * f, 1.f), es), fx_double(fx_join_wide(c[t], 2 * f + 1, 1.f), es));
              sum[t][f] = s0 ? cadd(sum[t][f], v) : v;
              if (cm && mag[f]) {
                const int e = (int)(em >> 20) + (int)(eb[f] >> 20), up = max(e, eref[t][f]);
                const float keep = spf_pow2(eref[t][f] - up), add = spf_pow2(e - up);
                tsum[t][f] = fmaf(tsum[t][f], keep, (ct[t][2 * f] + ct[t][2 * f + 1]) * add);
                bsum[t][f] = fmaf(bsum[t][f], keep, add);
                eref[t][f] = up;
              }
            }
          }
        }
      }
      __syncthreads();   // colmag, scale and W are read
    }
    if (half)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          other[warp & 3][t][f][lane] = nsteps ? sum[t][f] : mkc(0, 0);
          S.tother[warp & 3][t][f][lane] = tsum[t][f];
        }
    __syncthreads();
    if (!half)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int f = 0; f < 2; ++f)
          if (j0 + 4 * t + q < n && row0 + lr + 8 * f < G) {
            const int row = row0 + lr + 8 * f, j1 = j0 + 4 * t + q;
            cplx v = nsteps ? cadd(sum[t][f], other[warp & 3][t][f][lane]) : mkc(0, 0);
            if (tsum[t][f] + S.tother[warp & 3][t][f][lane] < FX_LOW * bsum[t][f]) {   // the element in FP64
              v = mkc(0, 0);
              for (int j = 0; j < ncols; ++j) cfma(v, col(j).x[row], col(j).rm[j1]);
            }
            put(row, j1, v);
          }
  next_pass:;
  }
}

__global__ void __launch_bounds__(SPF_THREADS) spf_drive_kernel(const SpfDesc* __restrict__ descs, int ndesc,
                                                                const SpfCol* __restrict__ cols,
                                                                cplx* __restrict__ out, cplx der) {
  extern __shared__ __align__(16) unsigned char spf_sm[];
  RowShared& S = *reinterpret_cast<RowShared*>(spf_sm);
  __shared__ SpfCol st[SPF_COLS];
  const SpfDesc& d = descs[warp_find_desc(descs, ndesc, (long long)blockIdx.x)];
  const SpfCol* gst = cols + d.col_first;
  const int ncols = d.col_count;
  // one chunk's columns in shared memory; longer lists are read where they are
  const bool local = ncols <= SPF_COLS;
  if (local && (int)threadIdx.x < ncols) st[threadIdx.x] = gst[threadIdx.x];
  __syncthreads();
  cplx* o = out + d.out_offset;
  const int G = d.G, row0 = (int)(blockIdx.x - d.block_start) * SPF_ROWS;
  const bool rot = der.x == 0.0 && der.y == -1.0, neg = der.x == -1.0 && der.y == 0.0;
  auto col = [&](int j) { return local ? st[j] : gst[j]; };
  stage_rows(S, 0, min(SPF_CHUNK, (ncols + 7) / 8), col, ncols, G, row0);
  row_products(S, ncols, col, d.n, G, row0, [&](int row, int j1, cplx v) {
    o[row + (long long)G * j1] = rot ? mkc(v.y, -v.x) : (neg ? mkc(-v.x, -v.y) : cmul(der, v));
  });
}

// (phi^H phi) X = phi^H dphi by Gauss-Jordan elimination of [S | O] without pivoting,
// which is stable for the Hermitian positive definite S.  Pivots are real; a thread
// holds EPT elements of get(row, column) in registers, and per pivot one column and one row pass through
// shared memory (two buffers, one barrier).  X transposed into Xt[j + n k] = X(k, j).
// Returns false at a pivot that is not positive.
template <int EPT, typename Get>
__device__ __forceinline__ bool solve_elimination(int n, Get&& get, cplx (*colb)[MAXN_SPF], cplx (*rowb)[2 * MAXN_SPF],
                                                  cplx* Xt) {
  cplx a[EPT];
  int ei[EPT], ec[EPT];   // the element's row and column (column -1: none)
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    const int e = threadIdx.x + q * SPF_THREADS;
    a[q] = mkc(0, 0);
    const int c = e / n, i = e - c * n;
    ei[q] = i;
    ec[q] = c < 2 * n ? c : -1;
    if (ec[q] < 0) continue;
    // the contraction's upper triangle is authoritative
    a[q] = c < n ? (i <= c ? get(i, c) : cconj(get(c, i))) : get(i, c);
    if (c == 0) colb[0][i] = a[q];
    if (i == 0) rowb[0][c] = a[q];
  }
  bool ok = true;
  for (int k = 0; k < n; ++k) {
    __syncthreads();
    const int b = k & 1;
    const double p = rowb[b][k].x;
    ok = ok && p > 0.0;
    const double pinv = newton_rcp(p);
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
      const int i = ei[q], c = ec[q];
      if (c <= k) continue;
      const cplx r = cscale(rowb[b][c], pinv);   // the scaled pivot row
      if (i == k) {
        a[q] = r;
      } else {
        const cplx f = colb[b][i];
        a[q].x = fma(-f.x, r.x, fma(f.y, r.y, a[q].x));
        a[q].y = fma(-f.x, r.y, fma(-f.y, r.x, a[q].y));
      }
      if (c == k + 1) colb[b ^ 1][i] = a[q];
      if (i == k + 1) rowb[b ^ 1][c] = a[q];
    }
  }
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    if (ec[q] >= n) Xt[ec[q] - n + n * ei[q]] = a[q];
  }
  return ok;
}

// Shared memory of the forms for n <= 8; in the first launch it takes the place of the
// matrix digits once these are read.
struct SpfSmall {
  cplx phs[8][SPF_PITCH], dph[8][SPF_PITCH];   // the CTA's rows of phi and dphi, zeros beyond G and n
  cplx so[128];                                // phi^H phi, then phi^H dphi ([j1 + 8 j2] each)
  cplx colb[2][MAXN_SPF], rowb[2][2 * MAXN_SPF], Xt[64];
  cplx red[4][128];                            // the warps' share of so
};
static_assert(sizeof(SpfSmall) <= sizeof(RowShared::W) && offsetof(SpfSmall, red) <= sizeof(RowShared::small),
              "takes the place of the digits, red alone that of the second warps' sums");

// so = (phi^H phi, phi^H dphi) of the CTA's 64 rows: warp w takes 16 rows of the first
// as in the contraction kernel for n <= 8, warp w + 4 of the second, sums that are small
// against the columns' largest elements again in FP64; the four warps' sums are added in
// order.
__device__ __forceinline__ void contract_rows(SpfSmall& T) {
  constexpr int NS = FX_NS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int which = warp >> 2, r0 = 16 * (warp & 3);
  const cplx (*Y)[SPF_PITCH] = which ? T.dph : T.phs;
  unsigned mx = 0u, my = 0u;
  cplx x[4], y[4];
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    x[f] = T.phs[g][r0 + 2 * q + (f & 1) + 8 * (f >> 1)];
    y[f] = Y[g][r0 + 2 * q + (f & 1) + 8 * (f >> 1)];
    mx = max(mx, fx_mag(x[f]));
    my = max(my, fx_mag(y[f]));
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    my = max(my, __shfl_xor_sync(0xffffffffu, my, o));
  }
  const unsigned ex = fx_ebits(mx), ey = fx_ebits(my);
  unsigned A[NS][4], B[NS][4];   // (re, im) of fibres 2 q, 2 q + 1, then of 2 q + 8, 2 q + 9
  unsigned ta[4], tb[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    unsigned s[NS];
    fx_digits(x[2 * h].x, x[2 * h + 1].x, ex, ex, s);
#pragma unroll
    for (int k = 0; k < NS; ++k) A[k][2 * h] = s[k];
    ta[2 * h] = fx_lead(s[0], s[1]);
    fx_digits(x[2 * h].y, x[2 * h + 1].y, ex, ex, s);
#pragma unroll
    for (int k = 0; k < NS; ++k) A[k][2 * h + 1] = s[k];
    ta[2 * h + 1] = fx_lead(s[0], s[1]);
    fx_digits(y[2 * h].x, y[2 * h + 1].x, ey, ey, s);
#pragma unroll
    for (int k = 0; k < NS; ++k) B[k][2 * h] = s[k];
    tb[h] = fx_lead(s[0], s[1]);
    fx_digits(y[2 * h].y, y[2 * h + 1].y, ey, ey, s);
#pragma unroll
    for (int k = 0; k < NS; ++k) B[k][2 * h + 1] = s[k];
    tb[h] = fx_add_half2(tb[h], fx_lead(s[0], s[1]));
  }
  float cr[NS][4], ci[NS][4], ct[4];
#pragma unroll
  for (int i = 0; i < NS; ++i)
#pragma unroll
    for (int j = 0; j + i < NS; ++j) {
      fx_mma16(cr[i + j], A[i], B[j][0], B[j][2], i == 0);   // the first product of weight i + j
      fx_mma16(ci[i + j], A[i], B[j][1], B[j][3], i == 0);
    }
  fx_mma16(ct, ta, tb[0], tb[1], true);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const unsigned es = fx_exp(ex, __shfl_sync(0xffffffffu, ey, 8 * q + 4 * i), 44);
    const unsigned wy = __shfl_sync(0xffffffffu, my, 8 * q + 4 * i);
    cplx v = mkc(fx_double(fx_join_wide(cr, i, 1.f) + fx_join_wide(ci, 2 + i, 1.f), es),
                 fx_double(fx_join_wide(ci, i, 1.f) - fx_join_wide(cr, 2 + i, 1.f), es));
    if (mx && wy && ct[i] + ct[2 + i] < FX_LOW) {
      v = mkc(0.0, 0.0);
      for (int r = 0; r < 16; ++r) cfma_conj(v, T.phs[g][r0 + r], Y[2 * q + i][r0 + r]);
    }
    T.red[warp & 3][64 * which + g + 8 * (2 * q + i)] = v;
  }
  const bool slow = __syncthreads_or(mx >= (FX_EMAX + 1u) << 20 || my >= (FX_EMAX + 1u) << 20);
  if (tid >= 128) return;
  cplx v = mkc(0.0, 0.0);
  if (slow) {
    const cplx* a = T.phs[tid & 7];
    const cplx* b = tid < 64 ? T.phs[tid >> 3] : T.dph[(tid - 64) >> 3];
    for (int r = 0; r < SPF_ROWS; ++r) cfma_conj(v, a[r], b[r]);
  } else {
#pragma unroll
    for (int w = 0; w < 4; ++w) v = cadd(v, T.red[w][tid]);
  }
  T.so[tid] = v;
}

// The next Runge-Kutta stage's input at element e: base + dt (sum_k c_k k_k + last v);
// stage_sum is the part that does not need v.
__device__ __forceinline__ cplx stage_sum(const SpfStage& g, long long e) {
  cplx s = mkc(0, 0);
  for (int k = 0; k < g.a.nk; ++k) {
    const cplx v = g.a.k[k][e];
    s.x = fma(g.a.c[k], v.x, s.x);
    s.y = fma(g.a.c[k], v.y, s.y);
  }
  return s;
}

// Solve from T.so and subtract the CTA's rows of phi X; with g.on also the next stage's
// input (the CTA's rows of phi are in shared memory by now, so it may replace them).  A
// thread has row threadIdx.x % 64 of columns threadIdx.x / 64 and + 4.  In FP64: eight
// instructions a row and column pair of warps.  Digit products were 2.4 us faster at n = 8
// and 400 points, but cut the rows of phi and X by their largest elements.
__device__ __forceinline__ bool solve_project(SpfSmall& T, const SpfDesc& d, int row0, cplx* o, const SpfStage& g) {
  const int n = d.n, G = d.G, row = threadIdx.x & (SPF_ROWS - 1), jr = threadIdx.x / SPF_ROWS;
  const bool in = row0 + row < G;
  cplx ss[2], bs[2];
  double dt = 0.0;
  if (g.on) {
    dt = g.dt_mode[g.elem_mode[d.out_offset - g.off]];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ss[i] = bs[i] = mkc(0.0, 0.0);
      if (in && jr + 4 * i < n) {
        const long long e = d.out_offset + row0 + row + (long long)G * (jr + 4 * i);
        ss[i] = stage_sum(g, e);
        bs[i] = g.base[e];
      }
    }
  }
  const bool ok = solve_elimination<1>(
      n, [&](int i, int c) { return c < n ? T.so[i + 8 * c] : T.so[64 + i + 8 * (c - n)]; }, T.colb, T.rowb, T.Xt);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int j = jr + 4 * i;
    if (!in || j >= n) break;
    cplx v = T.dph[j][row];
    for (int k = 0; k < n; ++k) {
      const cplx x = T.phs[k][row], c = T.Xt[j + n * k];
      v.x = fma(-x.x, c.x, fma(x.y, c.y, v.x));
      v.y = fma(-x.x, c.y, fma(-x.y, c.x, v.y));
    }
    const long long e = row0 + row + (long long)G * j;
    o[e] = v;
    if (g.on) {
      const cplx s = mkc(fma(g.last, v.x, ss[i].x), fma(g.last, v.y, ss[i].y));
      g.out[d.out_offset + e] = mkc(fma(dt, s.x, bs[i].x), fma(dt, s.y, bs[i].y));
    }
  }
  return ok;
}

// n <= 8.  ONE: every mode has at most 64 grid points, the CTA goes on to the solve.
// Otherwise dphi goes to out and the contractions of the CTA's rows to part.
template <bool ONE>
__global__ void __launch_bounds__(SPF_THREADS) spf_drive8_kernel(const SpfDesc* __restrict__ descs, int ndesc,
                                                                 const SpfCol* __restrict__ cols, cplx* out, cplx der,
                                                                 cplx* __restrict__ part, int* status, SpfStage g) {
  extern __shared__ __align__(16) unsigned char spf_sm[];
  RowShared& S = *reinterpret_cast<RowShared*>(spf_sm);
  SpfSmall& T = *reinterpret_cast<SpfSmall*>(&S.W);
  __shared__ SpfCol st[SPF_COLS];
  const SpfDesc& d = descs[warp_find_desc(descs, ndesc, (long long)blockIdx.x)];
  const SpfCol* gst = cols + d.col_first;
  const int ncols = d.col_count, n = d.n;
  // one chunk's columns in shared memory; longer lists are read where they are
  const bool local = ncols <= SPF_COLS;
  if (local && (int)threadIdx.x < ncols) st[threadIdx.x] = gst[threadIdx.x];
  __syncthreads();
  cplx* o = out + d.out_offset;
  const int G = d.G, row0 = (int)(blockIdx.x - d.block_start) * SPF_ROWS;
  const int row = threadIdx.x & (SPF_ROWS - 1), jr = threadIdx.x / SPF_ROWS;
  const bool rot = der.x == 0.0 && der.y == -1.0, neg = der.x == -1.0 && der.y == 0.0;
  auto col = [&](int j) { return local ? st[j] : gst[j]; };
  stage_rows(S, 0, min(SPF_CHUNK, (ncols + 7) / 8), col, ncols, G, row0);
  cplx ph[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    ph[i] = row0 + row < G && jr + 4 * i < n ? d.phi[row0 + row + (long long)G * (jr + 4 * i)] : mkc(0.0, 0.0);
  row_products(S, ncols, col, n, G, row0, [&](int r, int j1, cplx v) {
    const cplx w = rot ? mkc(v.y, -v.x) : (neg ? mkc(-v.x, -v.y) : cmul(der, v));
    T.dph[j1][r - row0] = w;
    if (!ONE) o[r + (long long)G * j1] = w;
  });
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    T.phs[jr + 4 * i][row] = ph[i];
    if (row0 + row >= G || jr + 4 * i >= n) T.dph[jr + 4 * i][row] = mkc(0.0, 0.0);
  }
  __syncthreads();
  contract_rows(T);
  if (!ONE) {
    if (threadIdx.x < 128) part[128LL * blockIdx.x + threadIdx.x] = T.so[threadIdx.x];   // the thread's own
    return;
  }
  __syncthreads();
  if (!solve_project(T, d, row0, o, g) && threadIdx.x == 0) atomicOr(status, DEVST_CHOL_FAIL);
}

// n <= 8, several CTAs per mode: every CTA adds its mode's contractions and solves for
// itself; its rows of phi and dphi are copied meanwhile.
__global__ void __launch_bounds__(SPF_THREADS) spf_project8_kernel(const SpfDesc* __restrict__ descs, int ndesc,
                                                                   cplx* out, const cplx* __restrict__ part,
                                                                   int* status, SpfStage g) {
  __shared__ SpfSmall T;
  const SpfDesc& d = descs[warp_find_desc(descs, ndesc, (long long)blockIdx.x)];
  const int n = d.n, G = d.G, tile = (int)(blockIdx.x - d.block_start), row0 = tile * SPF_ROWS;
  const int row = threadIdx.x & (SPF_ROWS - 1);
  cplx* o = out + d.out_offset;
  for (int j = threadIdx.x / SPF_ROWS; j < n && row0 + row < G; j += SPF_THREADS / SPF_ROWS) {
    copy_async16(&T.phs[j][row], d.phi + row0 + row + (long long)G * j);
    copy_async16(&T.dph[j][row], o + row0 + row + (long long)G * j);
  }
  if (threadIdx.x < 128) {
    cplx v = mkc(0.0, 0.0);
    const cplx* p = part + 128LL * d.block_start + threadIdx.x;
    const int ntile = (G + SPF_ROWS - 1) / SPF_ROWS;
#pragma unroll 4
    for (int t = 0; t < ntile; ++t) v = cadd(v, p[128LL * t]);
    T.so[threadIdx.x] = v;
  }
  copy_async_wait();
  __syncthreads();
  if (!solve_project(T, d, row0, o, g) && threadIdx.x == 0 && tile == 0) atomicOr(status, DEVST_CHOL_FAIL);
}
__global__ void __launch_bounds__(SPF_THREADS) spf_project_kernel(const SpfDesc* __restrict__ descs, int ndesc,
                                                                  cplx* __restrict__ out, int* status) {
  extern __shared__ __align__(16) unsigned char spf_sm[];
  RowShared& S = *reinterpret_cast<RowShared*>(spf_sm);
  __shared__ cplx colb[2][MAXN_SPF], rowb[2][2 * MAXN_SPF];
  const SpfDesc& d = descs[warp_find_desc(descs, ndesc, (long long)blockIdx.x)];
  const int n = d.n, G = d.G, tile = (int)(blockIdx.x - d.block_start), row0 = tile * SPF_ROWS;
  cplx* Xt = reinterpret_cast<cplx*>(spf_sm + sizeof(RowShared));   // [n][n]
  cplx* dph = Xt + n * n;                                           // [n][SPF_ROWS]
  cplx* o = out + d.out_offset;
  const cplx* phi = d.phi;
  auto col = [&](int j) { return SpfCol{phi + (long long)G * j, Xt + n * j}; };
  stage_rows(S, 0, (n + 7) / 8, col, n, G, row0);
  for (int e = threadIdx.x; e < n * SPF_ROWS; e += SPF_THREADS)
    if (row0 + (e & (SPF_ROWS - 1)) < G) copy_async16(dph + e, o + row0 + (e & (SPF_ROWS - 1)) + (long long)G * (e / SPF_ROWS));
  auto get = [&](int i, int c) { return c < n ? d.S[i + n * c] : d.O[i + n * (c - n)]; };
  const bool ok = n <= 8 ? solve_elimination<1>(n, get, colb, rowb, Xt)
                         : (n <= 16 ? solve_elimination<2>(n, get, colb, rowb, Xt) : solve_elimination<8>(n, get, colb, rowb, Xt));
  if (threadIdx.x == 0 && tile == 0 && !ok) atomicOr(status, DEVST_CHOL_FAIL);
  __syncthreads();
  row_products(S, n, col, n, G, row0, [&](int row, int j1, cplx v) {
    o[row + (long long)G * j1] = csub(dph[row - row0 + SPF_ROWS * j1], v);
  });
}

int launch_spf(const SpfDesc* d_descs, int ndesc, long long ntiles, int maxn, const SpfCol* d_cols,
               const HoleLaunch& holes, cplx* part, cplx* out, cplx der_factor, int* d_status, cudaStream_t st,
               const SpfStage& stage) {
  if (ndesc <= 0) return 0;
  const int smem = (int)sizeof(RowShared), smem_x = smem + (int)sizeof(cplx) * maxn * (maxn + SPF_ROWS);
  const unsigned nb = (unsigned)ntiles;
  if (maxn <= 8 && ntiles == ndesc) {
    spf_drive8_kernel<true><<<nb, SPF_THREADS, smem, st>>>(d_descs, ndesc, d_cols, out, der_factor, part, d_status, stage);
    return 1;
  }
  if (maxn <= 8) {
    spf_drive8_kernel<false><<<nb, SPF_THREADS, smem, st>>>(d_descs, ndesc, d_cols, out, der_factor, part, d_status, stage);
    spf_project8_kernel<<<nb, SPF_THREADS, 0, st>>>(d_descs, ndesc, out, part, d_status, stage);
    return 2;
  }
  spf_drive_kernel<<<nb, SPF_THREADS, smem, st>>>(d_descs, ndesc, d_cols, out, der_factor);
  launch_hole_fx(holes, st, 0, out);
  spf_project_kernel<<<nb, SPF_THREADS, smem_x, st>>>(d_descs, ndesc, out, d_status);
  return 3;
}

cudaError_t configure_spf() {
  cudaError_t e = allow_smem(spf_drive_kernel, sizeof(RowShared));
  if (e == cudaSuccess) e = allow_smem(spf_drive8_kernel<true>, sizeof(RowShared));
  if (e == cudaSuccess) e = allow_smem(spf_drive8_kernel<false>, sizeof(RowShared));
  if (e == cudaSuccess)
    e = allow_smem(spf_project_kernel, sizeof(RowShared) + sizeof(cplx) * MAXN_SPF * (MAXN_SPF + SPF_ROWS));
  return e;
}
