// Mode products and single-hole contractions of FP64 accuracy as exact digit
// products on the tensor cores (fixed.cuh) for sm_103a: precision 0, and the
// compensated products and contractions of the split modes.
#include <algorithm>

#include "kernels.cuh"
#include "fixed.cuh"

static int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 152;
  }();
  return n;
}

// ---------------------------------------------------------------------------
// Batched mode product (Mult_HeM_MatV / Mult_GM_MatV, gmctdh_objects.f90:1407-1468)
// A warp owns 16 fibres (l, :, r) (the rows of the MMA), the columns are the (re, im)
// of four outputs j'; a lane loads elements j = q, q + 4, .. of fibres g and g + 8 and
// receives outputs q, q + 4, .. of the same fibres, so neither side passes through
// shared memory.  A fibre shares one exponent, a matrix row another; eight digits of
// either, the 36 digit products of weight above 2^-64.  Bound by instruction issue:
// cutting digits and joining sums (about 50 instructions per complex element), not
// by the MMAs.
// ---------------------------------------------------------------------------

// The same product in FP64, for fibres or matrices outside the exponent range.
static __device__ __noinline__ void prod_fibre_fp64(const ProdDesc& d, long long l, long long r) {
  const long long L = d.L;
  for (int jo = 0; jo < d.nout; ++jo) {
    cplx acc = mkc(0.0, 0.0);
    for (int j = 0; j < d.nin; ++j) {
      const cplx m = d.conjT ? cconj(d.M[j + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * j];
      cfma(acc, m, load_c(d.X, l + L * (j + (long long)d.nin * r), d.xfmt));
    }
    cplx v = cmul(d.alpha, acc);
    cplx* y = d.Y + l + L * (jo + (long long)d.nout * r);
    if (d.accumulate) v = cadd(v, *y);
    *y = v;
  }
}
#define PROD_THREADS 128
#define PROD_NS 8
// resident CTAs per SM the register budget is set for
template <int NJ>
constexpr int prod_ctas() {
  return NJ <= 1 ? 5 : (NJ == 2 ? 4 : (NJ <= 4 ? 3 : 2));
}
// NJ: groups of four j.  The CTAs share the batch's fibres evenly, each walking a
// contiguous run (its matrix digits are cut once per descriptor, the next fibres'
// loads are in flight during the products).  split: few fibres in the batch -- a unit
// is 16 fibres and the four warps share the output groups, else 64 fibres.
template <int NJ>
__global__ void __launch_bounds__(PROD_THREADS, prod_ctas<NJ>())
    prod_fx_kernel(const ProdDesc* __restrict__ descs, int ndesc, long long nblocks, int split) {
  constexpr int NS = PROD_NS;
  constexpr int NK = (NJ + 1) / 2;            // k steps of 8 j; the last one of 4 for odd NJ
  constexpr bool BIG = NJ > 4;                // |D| may pass 2^22
  extern __shared__ uint2 Ws[];               // [NJ out groups][NK][NS][32]
  __shared__ unsigned rowexp[4 * NJ];         // exponent bits of the matrix rows
  __shared__ int s_bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int upb = split ? 8 : 2, ufib = split ? 16 : 64;   // units per 128-fibre block, fibres per unit
  const long long nunits = upb * nblocks;
  long long u0 = nunits * blockIdx.x / gridDim.x;
  const long long uend = nunits * (blockIdx.x + 1) / gridDim.x;
  int di = warp_find_desc(descs, ndesc, u0 / upb);
  for (; u0 < uend; ++di) {
    const ProdDesc& d = descs[di];
    const int nin = d.nin, nout = d.nout;
    const unsigned L = (unsigned)d.L;
    const unsigned nfib = (unsigned)(d.L * d.R);        // below 2^31
    const long long us = upb * d.block_start;
    const long long dend = min(uend, us + upb * (long long)((nfib + PROD_THREADS - 1) / PROD_THREADS));
    const int nt = (nout + 3) >> 2;
    const cplx* Xp = d.X + (long long)L * q;
    cplx* Yp = d.Y + (long long)L * q;
    const long long s4 = 4LL * L;                       // four j on
    const unsigned dl = ufib % L, dr = ufib / L;
    const long long Lx = d.L * (nin - 1), Ly = d.L * (nout - 1);
    unsigned p = (unsigned)(u0 - us) * ufib + (split ? 0 : warp * 16) + g, l[2], r[2];
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      r[f] = (p + 8 * f) / L;
      l[f] = p + 8 * f - L * r[f];
    }
    unsigned left = (unsigned)(dend - u0);
    cplx x[2][NJ];
    // element offset of fibre (l, r): l + L n r = p + L (n - 1) r
    auto fetch = [&]() {
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const cplx* xp = Xp + ((long long)(p + 8 * f) + Lx * r[f]);
        const bool act = p + 8 * f < nfib;
#pragma unroll
        for (int k = 0; k < NJ; ++k) {
          x[f][k] = mkc(0.0, 0.0);
          if (act && 4 * k + q < nin) x[f][k] = *xp;
          xp += s4;
        }
      }
    };
    fetch();
    __syncthreads();
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    for (int t = warp; t < nt; t += 4) {
      cplx mv[NJ];
      unsigned mag = 0;
      const int jo = 4 * t + (g >> 1);
#pragma unroll
      for (int k = 0; k < NJ; ++k) {
        const int j = 4 * k + q;
        mv[k] = mkc(0.0, 0.0);
        if (jo < nout && j < nin) mv[k] = d.conjT ? cconj(d.M[j + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * j];
        mag = max(mag, fx_mag(mv[k]));
      }
      mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 1));
      mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 2));
      if (!fx_ok(mag)) s_bad = 1;
      const unsigned eb = fx_ebits(mag);
      if (q == 0) rowexp[jo] = eb;
#pragma unroll
      for (int kk = 0; kk < NK; ++kk) {
        unsigned s0[NS], s1[NS];
        // column re: (Mr, -Mi); column im: (Mi, Mr)
        fx_digits<NS>(mv[2 * kk].x, mv[2 * kk].y, eb, eb, s0);
        if (2 * kk + 1 < NJ) fx_digits<NS>(mv[2 * kk + 1 < NJ ? 2 * kk + 1 : 0].x, mv[2 * kk + 1 < NJ ? 2 * kk + 1 : 0].y, eb, eb, s1);
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          const unsigned w0 = (g & 1) ? __byte_perm(s0[i], s0[i], 0x1032) : s0[i] ^ 0x80000000u;
          const unsigned w1 = 2 * kk + 1 < NJ ? ((g & 1) ? __byte_perm(s1[i], s1[i], 0x1032) : s1[i] ^ 0x80000000u) : 0u;
          Ws[((t * NK + kk) * NS + i) * 32 + lane] = make_uint2(w0, w1);
        }
      }
    }
    __syncthreads();
    const bool badM = s_bad;
    const bool plain = !d.accumulate && __double2hiint(d.alpha.x) == 0x3ff00000 && __double2loint(d.alpha.x) == 0 &&
                       (__double2hiint(d.alpha.y) << 1 | __double2loint(d.alpha.y)) == 0;   // alpha = 1
    for (; left; --left) {
      if (p - g >= nfib) break;
      int ef[2];
      bool bad = badM;
      unsigned A[NK][NS][4];   // digits: (fibre g, j), (fibre g + 8, j), (g, j + 4), (g + 8, j + 4)
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        unsigned mag = 0u;
#pragma unroll
        for (int k = 0; k < NJ; ++k) mag = max(mag, fx_mag(x[f][k]));
        mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 1));
        mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 2));
        bad = bad || !fx_ok(mag);
        const unsigned eb = fx_ebits(mag);
        ef[f] = (int)eb - ((2044 + 12 + 44) << 20);
#pragma unroll
        for (int k = 0; k < NJ; ++k) {
          unsigned s[NS];
          fx_digits<NS>(x[f][k].x, x[f][k].y, eb, eb, s);
#pragma unroll
          for (int i = 0; i < NS; ++i) A[k / 2][i][(k & 1) * 2 + f] = s[i];
        }
      }
      cplx* y[2];
#pragma unroll
      for (int f = 0; f < 2; ++f) y[f] = Yp + ((long long)(p + 8 * f) + Ly * r[f]);
      const bool any = __any_sync(0xffffffffu, bad);
      const bool act[2] = {p < nfib, p + 8 < nfib};
      const unsigned pp = p;
      p += ufib;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        l[f] += dl;
        r[f] += dr;
        if (l[f] >= L) { l[f] -= L; r[f] += 1; }
      }
      if (left > 1) fetch();
      if (any) {   // the warp's fibres in FP64
        if (q == 0 && (!split || warp == 0))
          for (int f = 0; f < 2; ++f)
            if (act[f]) prod_fibre_fp64(d, (pp + 8 * f) % L, (pp + 8 * f) / L);
        continue;
      }
#pragma unroll
      for (int t = 0; t < NJ; ++t) {
        if (t < nt && (!split || (t & 3) == warp)) {
          float c[NS][4];
#pragma unroll
          for (int kk = 0; kk < NK; ++kk) {
            if (kk == 0 || 8 * kk < nin) {
#pragma unroll
              for (int i = 0; i < NS; ++i) {
                const uint2 w = Ws[((t * NK + kk) * NS + i) * 32 + lane];
#pragma unroll
                for (int j = 0; j + i < NS; ++j) {
                  if (2 * kk + 1 < NJ) fx_mma16(c[i + j], A[kk][j], w.x, w.y, kk == 0 && i == 0);
                  else fx_mma8(c[i + j], A[kk][j], w.x, kk == 0 && i == 0);
                }
              }
            }
          }
          const int em = (int)rowexp[4 * t + q];
          if (4 * t + q < nout) {
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              const int es = em + ef[f];
              cplx v = mkc(fx_double(BIG ? fx_join_wide<NS, 0>(c, 2 * f) : fx_join<NS>(c, 2 * f), es),
                           fx_double(BIG ? fx_join_wide<NS, 0>(c, 2 * f + 1) : fx_join<NS>(c, 2 * f + 1), es));
              if (!plain) {
                v = cmul(d.alpha, v);
                if (d.accumulate && act[f]) v = cadd(v, y[f][t * s4]);
              }
              if (act[f]) y[f][t * s4] = v;
            }
          }
        }
      }
    }
    u0 = dend;
  }
}

template <int NJ>
static void prod_fx_go(const ProdDesc* d, int nd, long long nblocks, int persist, cudaStream_t st) {
  constexpr int smem = NJ * ((NJ + 1) / 2) * PROD_NS * 32 * (int)sizeof(uint2);
  static const cudaError_t configured =
      cudaFuncSetAttribute(prod_fx_kernel<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  (void)configured;
  long long most = (long long)sm_count() * prod_ctas<NJ>();
  // below one 64-fibre unit per SM the latency of a unit counts, not its cost
  const int split = 2 * nblocks < sm_count();
  if (persist > 0) most = std::min<long long>(most, persist);
  prod_fx_kernel<NJ><<<(unsigned)std::min((split ? 8 : 2) * nblocks, most), PROD_THREADS, smem, st>>>(d, nd, nblocks, split);
}

void launch_prod_fx(const ProdDesc* d, int nd, long long nblocks, int maxn, cudaStream_t st, int persist) {
  if (maxn <= 4) prod_fx_go<1>(d, nd, nblocks, persist, st);
  else if (maxn <= 8) prod_fx_go<2>(d, nd, nblocks, persist, st);
  else if (maxn <= 12) prod_fx_go<3>(d, nd, nblocks, persist, st);
  else if (maxn <= 16) prod_fx_go<4>(d, nd, nblocks, persist, st);
  else if (maxn <= 24) prod_fx_go<6>(d, nd, nblocks, persist, st);
  else prod_fx_go<8>(d, nd, nblocks, persist, st);
}

// ---------------------------------------------------------------------------
// Batched single-hole contraction, first stage (zher2k / zgemm('T','N') loops of
// Calc_rho1mode and Calc_MeanField, gmctdh_objects.f90:452-457, :595-600).
// Block b of a descriptor handles a contiguous share of the fibres.  A warp task is
// an 8 x 8 block of (j1, j2) pairs over every FS-th group of 16 fibres: the MMA's rows
// are (re, im) of eight X columns, its columns the re, then the im of eight Y columns,
// its inner dimension the fibres; lanes load what they hold, nothing is staged.  A
// column has one exponent, the largest so far in the task; when it grows, the sums so
// far go to FP64.  Seven digits (the operands rounded at 2^-54 of the column's largest
// element), the 34 digit products of weight above 2^-64.  The last block of a
// descriptor to finish adds the blocks' partials in block order into the first.
// ---------------------------------------------------------------------------
#define HOLE_NS 7        // digits per operand
#define HOLE_ND 8        // weights kept
#define HOLE_FLUSH 8     // groups of 16 fibres between flushes: 128 x 6 x 2^14 < 2^24
#define HOLE_WARPS 4
#define HOLE_MTHREADS (32 * HOLE_WARPS)

// 1 x 1 contractions (inner products): every thread strides over elements with
// coalesced loads, the block reduces in shared memory.
static __device__ void dot_block(const HoleDesc& d, int b, cplx* red) {
  const long long n = d.L * d.R;
  const int tid = threadIdx.x;
  cplx acc = mkc(0, 0);
  for (long long i = (long long)b * HOLE_MTHREADS + tid; i < n; i += (long long)d.nblk * HOLE_MTHREADS)
    cfma_conj(acc, load_c(d.X, i, d.xfmt), load_c(d.Y, i, d.yfmt));
  red[tid] = acc;
  __syncthreads();
  for (int s = HOLE_MTHREADS / 2; s > 0; s >>= 1) {
    if (tid < s) red[tid] = cadd(red[tid], red[tid + s]);
    __syncthreads();
  }
  if (tid == 0) d.partial[b] = red[0];
}

// The block's contraction in FP64 from global memory, for operands outside the
// exponent range (fibres p0 .. p1).
static __device__ __noinline__ void hole_block_fp64(const HoleDesc& d, const cplx* Y, int b, unsigned p0, unsigned p1) {
  const long long L = d.L;
  for (int pr = threadIdx.x; pr < d.n1 * d.n2; pr += blockDim.x) {
    const int j1 = pr % d.n1, j2 = pr / d.n1;
    cplx acc = mkc(0, 0);
    for (long long p = p0; p < p1; ++p) {
      const long long r = p / L, l = p - r * L;
      cfma_conj(acc, load_c(d.X, l + L * (j1 + (long long)d.n1 * r), d.xfmt),
                load_c(Y, l + L * (j2 + (long long)d.n2 * r), d.yfmt));
    }
    d.partial[(long long)b * d.n1 * d.n2 + pr] = acc;
  }
}

// F32: operands may be complex FP32
template <bool F32>
__device__ __forceinline__ void hole_fx_block(const HoleDesc& d, int b, const cplx* ybase) {
  constexpr int NS = HOLE_NS, ND = HOLE_ND;
  extern __shared__ cplx red[];   // [pair blocks][FS][64]
  __shared__ int s_slow;
  const cplx* Yp = d.Y ? d.Y : ybase + d.yoff;
  const int n1 = d.n1, n2 = d.n2, npairs = n1 * n2;
  if (npairs == 1 && d.Y && d.L * d.R >= HOLE_MTHREADS) {
    dot_block(d, b, red);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int xfmt = F32 ? d.xfmt : 0, yfmt = F32 ? d.yfmt : 0;
  // X = Y (density matrices, SPF overlaps): C is Hermitian, only the blocks on and
  // above the diagonal are computed
  const bool sym = d.X == d.Y && n1 == n2 && d.xfmt == d.yfmt;
  const int b1 = (n1 + 7) >> 3, b2 = (n2 + 7) >> 3;
  const int nbp = sym ? b1 * (b1 + 1) / 2 : b1 * b2;
  const int FS = (nbp & 3) == 0 ? 1 : ((nbp & 1) == 0 ? 2 : 4);   // tasks fill the warps
  const unsigned L = (unsigned)d.L, nfib = (unsigned)(d.L * d.R);
  const unsigned ngrp = (nfib + 15) / 16;
  const unsigned g0 = (unsigned)((unsigned long long)ngrp * b / d.nblk);
  const unsigned g1 = (unsigned)((unsigned long long)ngrp * (b + 1) / d.nblk);
  const unsigned dl = (16u * FS) % L, dr = (16u * FS) / L;
  if (tid == 0) s_slow = 0;
  __syncthreads();
  bool slow = false;
  for (int task = warp; task < nbp * FS; task += HOLE_WARPS) {
    const int pb = task / FS, fs = task - pb * FS;
    int c1 = pb % b1, c2 = pb / b1;
    if (sym) {   // pb -> (c1 <= c2), c2-major
      int rem = pb;
      c2 = 0;
      while (rem > c2) rem -= ++c2;
      c1 = rem;
    }
    const bool same = sym && c1 == c2;
    const int jx = 8 * c1 + g, jy = 8 * c2 + g;   // the lane's columns
    // the lane's fibres of a group: 2 q, 2 q + 1, 2 q + 8, 2 q + 9
    unsigned p = 16u * (g0 + fs) + 2 * q, l[4], r[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const unsigned pf = p + (f & 1) + 8 * (f >> 1);
      r[f] = pf / L;
      l[f] = pf - L * r[f];
    }
    cplx x[4], y[4];
    auto fetch = [&]() {
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const bool in = p + (f & 1) + 8 * (f >> 1) < nfib;
        x[f] = y[f] = mkc(0.0, 0.0);
        if (in && jx < n1) x[f] = load_c(d.X, l[f] + (long long)L * (jx + (long long)n1 * r[f]), xfmt);
        if (!same && in && jy < n2) y[f] = load_c(Yp, l[f] + (long long)L * (jy + (long long)n2 * r[f]), yfmt);
        l[f] += dl;
        r[f] += dr;
        if (l[f] >= L) { l[f] -= L; r[f] += 1; }
      }
      p += 16 * FS;
    };
    float cr[ND][4], ci[ND][4];   // sums with Yr and Yi: rows Xr (0, 1), Xi (2, 3)
#pragma unroll
    for (int k = 0; k < ND; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) cr[k][i] = ci[k][i] = 0.f;
    cplx acc[2] = {mkc(0.0, 0.0), mkc(0.0, 0.0)};
    constexpr unsigned emin = (unsigned)FX_EMIN << 20;
    unsigned ex = emin, ey = emin;
    int pend = 0;
    bool fresh = true;
    auto flush = [&]() {
      // conj(x) y = (Xr Yr + Xi Yi) + i (Xr Yi - Xi Yr) of columns 2 q, 2 q + 1
      const unsigned e2[2] = {__shfl_sync(0xffffffffu, same ? ex : ey, 8 * q), __shfl_sync(0xffffffffu, same ? ex : ey, 8 * q + 4)};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const long long re = fx_join_wide<ND, 1>(cr, i) + fx_join_wide<ND, 1>(ci, 2 + i);
        const long long im = fx_join_wide<ND, 1>(ci, i) - fx_join_wide<ND, 1>(cr, 2 + i);
        const int es = (int)(ex + e2[i]) - ((2044 + 12 + 43) << 20);
        const cplx v = mkc(fx_double(re, es), fx_double(im, es));
        acc[i] = fresh ? v : cadd(acc[i], v);
      }
#pragma unroll
      for (int k = 0; k < ND; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) cr[k][i] = ci[k][i] = 0.f;
      fresh = false;
      pend = 0;
    };
    fetch();
    for (unsigned gr = g0 + fs; gr < g1; gr += FS) {
      unsigned mx = max(max(fx_mag(x[0]), fx_mag(x[1])), max(fx_mag(x[2]), fx_mag(x[3])));
      unsigned my = max(max(fx_mag(y[0]), fx_mag(y[1])), max(fx_mag(y[2]), fx_mag(y[3])));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      my = max(my, __shfl_xor_sync(0xffffffffu, my, 1));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      my = max(my, __shfl_xor_sync(0xffffffffu, my, 2));
      // out of range, or tiny with nothing larger in the column before it
      slow = slow || (!fx_ok(mx) && (mx >= emin || ex == emin)) ||
             (!fx_ok(my) && (my >= emin || ey == emin));
      const bool grow = mx >= ex + (1u << 20) || my >= ey + (1u << 20);
      if (__any_sync(0xffffffffu, grow) || pend == HOLE_FLUSH) {
        if (pend) flush();
        ex = max(ex, mx & FX_EBITS);
        ey = max(ey, my & FX_EBITS);
      }
      unsigned A[NS][4], Br[NS][2], Bi[NS][2];
      {
        unsigned s[NS];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          fx_digits<NS>(x[2 * h].x, x[2 * h + 1].x, ex, ex, s);
#pragma unroll
          for (int k = 0; k < NS; ++k) A[k][2 * h] = s[k];
          fx_digits<NS>(x[2 * h].y, x[2 * h + 1].y, ex, ex, s);
#pragma unroll
          for (int k = 0; k < NS; ++k) A[k][2 * h + 1] = s[k];
        }
        if (same) {
#pragma unroll
          for (int k = 0; k < NS; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              Br[k][h] = A[k][2 * h];
              Bi[k][h] = A[k][2 * h + 1];
            }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            fx_digits<NS>(y[2 * h].x, y[2 * h + 1].x, ey, ey, s);
#pragma unroll
            for (int k = 0; k < NS; ++k) Br[k][h] = s[k];
            fx_digits<NS>(y[2 * h].y, y[2 * h + 1].y, ey, ey, s);
#pragma unroll
            for (int k = 0; k < NS; ++k) Bi[k][h] = s[k];
          }
        }
      }
      if (gr + FS < g1) fetch();
#pragma unroll
      for (int i = 0; i < NS; ++i)
#pragma unroll
        for (int j = 0; j < NS && j + i < ND; ++j) {
          fx_mma16(cr[i + j], A[i], Br[j][0], Br[j][1], false);
          fx_mma16(ci[i + j], A[i], Bi[j][0], Bi[j][1], false);
        }
      ++pend;
    }
    if (pend) flush();
    // (j1, j2) = (g, 2 q), (g, 2 q + 1) of the task's block
    red[(pb * FS + fs) * 64 + g + 8 * (2 * q)] = acc[0];
    red[(pb * FS + fs) * 64 + g + 8 * (2 * q + 1)] = acc[1];
  }
  if (slow) s_slow = 1;
  __syncthreads();
  if (s_slow) {
    hole_block_fp64(d, Yp, b, 16u * g0, min(16u * g1, nfib));
    return;
  }
  cplx* out = d.partial + (long long)b * npairs;
  for (int pr = tid; pr < npairs; pr += HOLE_MTHREADS) {
    int j1 = pr % n1, j2 = pr / n1;
    const bool lower = sym && (j1 >> 3) > (j2 >> 3);   // conj of the transposed pair
    if (lower) { const int tmp = j1; j1 = j2; j2 = tmp; }
    const int c1 = j1 >> 3, c2 = j2 >> 3, pb = sym ? c2 * (c2 + 1) / 2 + c1 : c1 + b1 * c2;
    const cplx* s = red + pb * FS * 64 + (j1 & 7) + 8 * (j2 & 7);
    cplx v = s[0];
    for (int k = 1; k < FS; ++k) v = cadd(v, s[64 * k]);
    out[pr] = lower ? cconj(v) : v;
  }
}

// The block that finishes last adds the descriptor's partials into the first, in
// block order, and resets the counter for the next launch.
static __device__ __forceinline__ void hole_sum_blocks(const HoleDesc& d) {
  __shared__ bool s_last;
  const int npairs = d.n1 * d.n2, nblk = d.nblk;
  if (nblk == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(d.counter, 1u) == (unsigned)(nblk - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int sub = 1;   // neighbouring threads per pair
  while (2 * sub * npairs <= HOLE_MTHREADS && 2 * sub <= min(nblk, 32)) sub *= 2;
  for (int w0 = 0; w0 < npairs * sub; w0 += HOLE_MTHREADS) {
    const int w = w0 + threadIdx.x, pr = w / sub, k0 = w - pr * sub;
    const bool on = pr < npairs;
    cplx s = mkc(0, 0);
    if (on)
      for (int k = k0; k < nblk; k += sub) s = cadd(s, __ldcg(d.partial + (long long)k * npairs + pr));
    for (int o = 1; o < sub; o <<= 1)
      s = cadd(s, mkc(__shfl_xor_sync(0xffffffffu, s.x, o), __shfl_xor_sync(0xffffffffu, s.y, o)));
    __syncwarp();
    if (on && k0 == 0) d.partial[pr] = s;
  }
  if (threadIdx.x == 0) *d.counter = 0u;
}

// CTA b takes the batch's blocks b, b + gridDim.x, ...: one each, or the persistent
// form (each block writes its own partial, so the sums do not depend on the grid).
template <bool F32>
__global__ void __launch_bounds__(HOLE_MTHREADS, 3)
    hole_fx_kernel(const HoleDesc* __restrict__ descs, int ndesc, long long nblocks, const cplx* ybase) {
  for (long long bb = blockIdx.x; bb < nblocks; bb += gridDim.x) {
    const HoleDesc& d = descs[warp_find_desc(descs, ndesc, bb)];
    if (bb != blockIdx.x) __syncthreads();   // the shared sums are rewritten
    hole_fx_block<F32>(d, (int)(bb - d.block_start), ybase);
    hole_sum_blocks(d);
  }
}

void launch_hole_fx(const HoleDesc* d, int nd, long long nblocks, int maxn, bool f32, cudaStream_t st, int persist,
                    const cplx* ybase) {
  // the most tasks (pair blocks x fibre shares) of any n1, n2 <= maxn: 1 x 4, 3 x 4, 9 x 4
  const int smem = (int)sizeof(cplx) * 64 * (maxn <= 8 ? 4 : (maxn <= 16 ? 12 : 36));
  const unsigned grid = (unsigned)(persist > 0 ? std::min<long long>(nblocks, persist) : nblocks);
  if (f32) hole_fx_kernel<true><<<grid, HOLE_MTHREADS, smem, st>>>(d, nd, nblocks, ybase);
  else hole_fx_kernel<false><<<grid, HOLE_MTHREADS, smem, st>>>(d, nd, nblocks, ybase);
}
