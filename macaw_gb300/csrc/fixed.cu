// Mode products and single-hole contractions of FP64 accuracy as exact digit
// products on the tensor cores (fixed.cuh) for sm_103a: precision 0, and the
// FP64-accurate products and contractions of the mixed modes.
#include <algorithm>

#include "kernels.cuh"
#include "fixed.cuh"

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
      unsigned ef[2];
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
        ef[f] = fx_exp(eb, 0u, 44);
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
          const unsigned em = rowexp[4 * t + q];
          if (4 * t + q < nout) {
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              const unsigned es = em + ef[f];
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
constexpr int prod_smem() {
  return NJ * ((NJ + 1) / 2) * PROD_NS * 32 * (int)sizeof(uint2);
}
template <int NJ>
static void prod_fx_go(const ProdDesc* d, int nd, long long nblocks, int persist, cudaStream_t st) {
  long long most = (long long)sm_count() * prod_ctas<NJ>();
  // below one 64-fibre unit per SM the latency of a unit counts, not its cost
  const int split = 2 * nblocks < sm_count();
  if (persist > 0) most = std::min<long long>(most, persist);
  prod_fx_kernel<NJ><<<(unsigned)std::min((split ? 8 : 2) * nblocks, most), PROD_THREADS, prod_smem<NJ>(), st>>>(d, nd, nblocks, split);
}

// The tcgen05 form (tc.cu) takes batches of 5 to 16 SPFs that give every one of its CTAs
// (four per SM up to 8 SPFs, two above) at least two tiles of 128 fibres, so that the
// matrix digits and the pipeline's start are paid for: 57 products of 32,768 fibres of 8
// took 191 us against 226, of 248,832 fibres of 12 2,206 against 2,900; a batch of 700
// tiles of 5 to 9 took 19 against 17.
void launch_prod_fx(const ProdDesc* d, int nd, long long nblocks, int maxn, int* status, cudaStream_t st, int persist) {
  if (persist <= 0 && tc_enabled() && maxn > 4 && maxn <= 16 && nblocks >= (maxn <= 8 ? 8 : 4) * (long long)sm_count()) {
    launch_prod_digits_tc(d, nd, nblocks, maxn, status, st);
    return;
  }
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
// Block b of a descriptor handles a contiguous share of the fibres.  For n1, n2 <= 8 a
// warp takes every fourth group of 16 fibres: the MMA's rows
// are (re, im) of eight X columns, its columns the re, then the im of eight Y columns,
// its inner dimension the fibres; lanes load what they hold, nothing is staged.  A
// column has one exponent, the largest so far in the warp; when it grows, the sums so
// far go to FP64.  Seven digits (the operands rounded at 2^-54 of the column's largest
// element), the 34 digit products of weight above 2^-64.  The last block of a
// descriptor to finish adds the blocks' partials in block order into the first.
// ---------------------------------------------------------------------------
#define HOLE_NS 7        // digits per operand
#define HOLE_ND 8        // weights kept
#define HOLE_FLUSH 8     // groups of 16 fibres between flushes: 128 x 6 x 2^14 < 2^24
#define HOLE_WARPS 4     // per block; twice as many where n1 or n2 is above eight

// 1 x 1 contractions (inner products): every thread strides over elements with
// coalesced loads, the block reduces in shared memory.
static __device__ void dot_block(const HoleDesc& d, int b, cplx* red) {
  constexpr int T = 32 * HOLE_WARPS;
  const long long n = d.L * d.R;
  const int tid = threadIdx.x;
  cplx acc = mkc(0, 0);
  for (long long i = (long long)b * T + tid; i < n; i += (long long)d.nblk * T)
    cfma_conj(acc, load_c(d.X, i, d.xfmt), load_c(d.Y, i, d.yfmt));
  red[tid] = acc;
  __syncthreads();
  for (int s = T / 2; s > 0; s >>= 1) {
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
  constexpr int NS = HOLE_NS, ND = HOLE_ND, W = HOLE_WARPS;
  extern __shared__ cplx red[];   // [warp][64]
  __shared__ int s_slow;
  const cplx* Yp = d.Y ? d.Y : ybase + d.yoff;
  const int n1 = d.n1, n2 = d.n2, npairs = n1 * n2;
  if (npairs == 1 && d.Y && d.L * d.R >= 32 * W) {
    dot_block(d, b, red);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int xfmt = F32 ? d.xfmt : 0, yfmt = F32 ? d.yfmt : 0;
  // X = Y (density matrices, SPF overlaps): the digits serve both operands
  const bool sym = d.X == d.Y && n1 == n2 && d.xfmt == d.yfmt;
  const unsigned L = (unsigned)d.L, nfib = (unsigned)(d.L * d.R);
  const unsigned ngrp = (nfib + 15) / 16;
  const unsigned g0 = (unsigned)((unsigned long long)ngrp * b / d.nblk);
  const unsigned g1 = (unsigned)((unsigned long long)ngrp * (b + 1) / d.nblk);
  const unsigned dl = (16u * W) % L, dr = (16u * W) / L;
  if (tid == 0) s_slow = 0;
  __syncthreads();
  bool slow = false;
  {
    const bool same = sym;
    const int jx = g, jy = g;   // the lane's columns
    // the lane's fibres of a group: 2 q, 2 q + 1, 2 q + 8, 2 q + 9
    unsigned p = 16u * (g0 + warp) + 2 * q, l[4], r[4];
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
      p += 16 * W;
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
        const unsigned es = fx_exp(ex, e2[i], 43);
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
    for (unsigned gr = g0 + warp; gr < g1; gr += W) {
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
      if (gr + W < g1) fetch();
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
    // (j1, j2) = (g, 2 q), (g, 2 q + 1)
    red[warp * 64 + g + 8 * (2 * q)] = acc[0];
    red[warp * 64 + g + 8 * (2 * q + 1)] = acc[1];
  }
  if (slow) s_slow = 1;
  __syncthreads();
  if (s_slow) {
    hole_block_fp64(d, Yp, b, 16u * g0, min(16u * g1, nfib));
    return;
  }
  cplx* out = d.partial + (long long)b * npairs;
  for (int pr = tid; pr < npairs; pr += 32 * W) {
    const cplx* s = red + pr % n1 + 8 * (pr / n1);
    cplx v = s[0];
    for (int k = 1; k < W; ++k) v = cadd(v, s[64 * k]);
    out[pr] = v;
  }
}

// The same for n1 or n2 above eight.  Tiles of two by two column blocks: each operand
// block of 32 fibres is cut once, by one warp, into shared memory in the order the MMAs
// read it (an uint4 per lane, digit and group of 16 fibres: re, im of fibres 2 q, 2 q + 1,
// then of 2 q + 8, 2 q + 9), and every warp takes a pair block of the tile.  Where every
// pair block cut its own operands, cutting bound the kernel (ALU 52 %, tensor pipe 36 %).
// A column block of at most four columns puts re and im side by side into one MMA.
// Warps 0-3 cut the next stage while warps 4-7 multiply this one: with every warp doing
// both in turn the phases of a block did not overlap.
// 42 contractions of 248,832 fibres, 12 x 12 each: 3,117 -> 2,295 us.
#define HOLEW_GRP 2      // groups of 16 fibres per stage
#define HOLEW_FLUSH (HOLE_FLUSH / HOLEW_GRP)
#define HOLEW_SLOTS 3    // stages of operands in flight
struct HoleWide {
  uint4 dig[2][4][HOLEW_GRP][HOLE_NS][32];   // [buffer][operand block][group][digit][lane]
  cplx raw[HOLEW_SLOTS][4][4 * HOLEW_GRP][32];  // operands: [slot][block][fibre of the lane][lane]
  cplx sum[4][64];
  unsigned ex[2][4][8];                      // the columns' exponents
  int grow[2][4];
  int slow;
};
// both roles pass the same barriers: one before the first stage, one after each
__device__ __forceinline__ void hole_stage_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(64 * HOLE_WARPS) : "memory");
}
template <bool F32>
__device__ __forceinline__ void hole_cut(HoleWide& sh, const HoleDesc& d, const cplx* Yp, bool& slow, bool cut, bool isx,
                                         int j0, unsigned nfib, unsigned g0, unsigned g1) {
  constexpr int NS = HOLE_NS, NP = 4 * HOLEW_GRP;   // fibres per lane and stage
  constexpr unsigned emin = (unsigned)FX_EMIN << 20;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const unsigned L = (unsigned)d.L, dl = (16u * HOLEW_GRP) % L, dr = (16u * HOLEW_GRP) / L;
  const cplx* P = isx ? d.X : Yp;
  const int np = isx ? d.n1 : d.n2, j = j0 + g;
  const int fmt = F32 ? (isx ? d.xfmt : d.yfmt) : 0;
  unsigned grp = g0, ec = emin, l[NP / 2], r[NP / 2];   // fibres 2 q (+ 8) of each group
#pragma unroll
  for (int h = 0; h < NP / 2; ++h) {
    const unsigned p = 16 * g0 + 8 * h + 2 * q;
    r[h] = p / L;
    l[h] = p - L * r[h];
  }
  const unsigned raw0 = (unsigned)__cvta_generic_to_shared(&sh.raw[0][warp][0][lane]);
  constexpr unsigned slot_bytes = sizeof(sh.raw[0]), point_bytes = sizeof(sh.raw[0][0][0]);
  auto copy = [&](unsigned dst, unsigned ll, unsigned rr, bool in) {
    const long long e = ll + (long long)L * (j + (long long)np * rr);
    if (F32 && fmt)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(reinterpret_cast<const float2*>(P) + (in ? e : 0)), "r"(in ? 8 : 0) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(P + (in ? e : 0)), "r"(in ? 16 : 0) : "memory");
  };
  int wslot = 0, rslot = 0;
  auto fetch = [&]() {   // the next stage's elements, each lane its own: nothing to synchronise
    if (cut && grp < g1) {
#pragma unroll
      for (int h = 0; h < NP / 2; ++h) {
        const unsigned p = 16 * grp + 8 * h + 2 * q;
        const bool in = j < np && grp + (h >> 1) < g1, wrap = l[h] + 1 == L;
        const unsigned dst = raw0 + wslot * slot_bytes + 2 * h * point_bytes;
        copy(dst, l[h], r[h], in && p < nfib);
        copy(dst + point_bytes, wrap ? 0u : l[h] + 1, wrap ? r[h] + 1 : r[h], in && p + 1 < nfib);
        l[h] += dl;
        r[h] += dr;
        if (l[h] >= L) { l[h] -= L; r[h] += 1; }
      }
    }
    grp += HOLEW_GRP;
    wslot = wslot + 1 == HOLEW_SLOTS ? 0 : wslot + 1;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto stage = [&](int buf) {   // cut the oldest stage in flight into buffer buf
    asm volatile("cp.async.wait_group %0;" ::"n"(HOLEW_SLOTS - 1) : "memory");
    cplx x[NP];
#pragma unroll
    for (int f = 0; f < NP; ++f) x[f] = load_c(&sh.raw[rslot][warp][f][lane], 0, fmt);
    rslot = rslot + 1 == HOLEW_SLOTS ? 0 : rslot + 1;
    unsigned m = 0u;
#pragma unroll
    for (int f = 0; f < NP; ++f) m = max(m, fx_mag(x[f]));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
    // out of range, or tiny with nothing larger in the column before it
    slow = slow || (!fx_ok(m) && (m >= emin || ec == emin));
    const bool grow = m >= ec + (1u << 20);
    if (grow) ec = m & FX_EBITS;
    const bool any = __any_sync(0xffffffffu, grow);
    if (lane == 0) sh.grow[buf][warp] = any;
    if (q == 0) sh.ex[buf][warp][g] = ec;
#pragma unroll
    for (int gg = 0; gg < HOLEW_GRP; ++gg) {
      unsigned s[4][NS];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        fx_digits<NS>(x[4 * gg + 2 * h].x, x[4 * gg + 2 * h + 1].x, ec, ec, s[2 * h]);
        fx_digits<NS>(x[4 * gg + 2 * h].y, x[4 * gg + 2 * h + 1].y, ec, ec, s[2 * h + 1]);
      }
#pragma unroll
      for (int k = 0; k < NS; ++k) sh.dig[buf][warp][gg][k][lane] = make_uint4(s[0][k], s[1][k], s[2][k], s[3][k]);
    }
  };
  for (int k = 0; k < HOLEW_SLOTS; ++k) fetch();
  if (cut) stage(0);
  fetch();
  hole_stage_barrier();
  int buf = 1;
  for (unsigned gr = g0; gr < g1; gr += HOLEW_GRP, buf ^= 1) {
    if (cut && gr + HOLEW_GRP < g1) stage(buf);
    fetch();
    hole_stage_barrier();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}
template <bool PACKED>
__device__ __forceinline__ void hole_mul_go(HoleWide& sh, cplx* acc, bool mine, int xb, int yb, int split, int half,
                                            unsigned g0, unsigned g1) {
  constexpr int NS = HOLE_NS, ND = HOLE_ND;
  constexpr unsigned emin = (unsigned)FX_EMIN << 20;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  float cr[ND][4], ci[ND][4];   // sums with Yr and Yi (packed: all in cr): rows Xr (0, 1), Xi (2, 3)
#pragma unroll
  for (int k = 0; k < ND; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) cr[k][i] = ci[k][i] = 0.f;
  unsigned e1 = emin, e2[2] = {emin, emin};
  int pend = 0;
  auto flush = [&]() {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned es = fx_exp(e1, e2[i], 43);
      const long long a = fx_join_wide<ND, 1>(cr, i), b = fx_join_wide<ND, 1>(cr, 2 + i);
      if (PACKED) {
        // conj(x) y of a column: re = Xr Yr + Xi Yi in lanes q < 2, im = Xr Yi - Xi Yr in q + 2
        const long long o = __shfl_xor_sync(0xffffffffu, b, 2);
        acc[i].x += fx_double(q < 2 ? a + o : a - o, es);
      } else {
        const long long re = a + fx_join_wide<ND, 1>(ci, 2 + i), im = fx_join_wide<ND, 1>(ci, i) - b;
        acc[i] = cadd(acc[i], mkc(fx_double(re, es), fx_double(im, es)));
      }
    }
#pragma unroll
    for (int k = 0; k < ND; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) cr[k][i] = ci[k][i] = 0.f;
    pend = 0;
  };
  hole_stage_barrier();
  int buf = 0;
  for (unsigned gr = g0; gr < g1; gr += HOLEW_GRP, buf ^= 1) {
    if (mine) {
      if (sh.grow[buf][xb] || sh.grow[buf][yb] || pend == HOLEW_FLUSH) {
        if (pend) flush();
        e1 = sh.ex[buf][xb][g];
        const int cy = PACKED ? 2 * (q & 1) : 2 * q;
        e2[0] = sh.ex[buf][yb][cy];
        e2[1] = sh.ex[buf][yb][cy + 1];
      }
#pragma unroll 1
      for (int gg = split == 2 ? half : 0; gg < HOLEW_GRP; gg += split) {
        unsigned A[NS][4];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
          const uint4 v = sh.dig[buf][xb][gg][k][lane];
          A[k][0] = v.x;
          A[k][1] = v.y;
          A[k][2] = v.z;
          A[k][3] = v.w;
        }
        // packed: columns g & 3, re for g < 4, im above
        const uint4* yd = &sh.dig[buf][yb][gg][0][PACKED ? lane & 15 : lane];
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          const uint4 v = yd[32 * j];
          if (PACKED) {
            const unsigned w0 = g < 4 ? v.x : v.y, w1 = g < 4 ? v.z : v.w;
#pragma unroll
            for (int i = 0; i < NS && i + j < ND; ++i) fx_mma16(cr[i + j], A[i], w0, w1, false);
          } else {
#pragma unroll
            for (int i = 0; i < NS && i + j < ND; ++i) {
              fx_mma16(cr[i + j], A[i], v.x, v.z, false);
              fx_mma16(ci[i + j], A[i], v.y, v.w, false);
            }
          }
        }
      }
      ++pend;
    }
    hole_stage_barrier();
  }
  if (pend) flush();
}
__device__ __forceinline__ void hole_mul(HoleWide& sh, cplx* acc, bool mine, bool packed, int xb, int yb, int split,
                                         int half, unsigned g0, unsigned g1) {
  if (packed) hole_mul_go<true>(sh, acc, mine, xb, yb, split, half, g0, g1);
  else hole_mul_go<false>(sh, acc, mine, xb, yb, split, half, g0, g1);
}
template <bool F32>
__device__ __forceinline__ void hole_wide_block(const HoleDesc& d, int b, const cplx* ybase, int nsm) {
  extern __shared__ cplx red[];
  HoleWide& sh = *reinterpret_cast<HoleWide*>(red);
  const cplx* Yp = d.Y ? d.Y : ybase + d.yoff;
  const int n1 = d.n1, n2 = d.n2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const bool sym = d.X == d.Y && n1 == n2 && d.xfmt == d.yfmt;
  const int b1 = (n1 + 7) >> 3, b2 = (n2 + 7) >> 3;
  const unsigned nfib = (unsigned)(d.L * d.R);
  const unsigned ngrp = (nfib + 15) / 16;
  const unsigned g0 = (unsigned)((unsigned long long)ngrp * b / d.nblk);
  const unsigned g1 = (unsigned)((unsigned long long)ngrp * (b + 1) / d.nblk);
  // the light pair blocks (short last column block) fall to other sub-partitions in
  // every other wave of CTAs
  const int vw = (warp + 2 * (int)((blockIdx.x / nsm) & 1)) & 3;
  cplx* out = d.partial + (long long)b * n1 * n2;
  if (tid == 0) sh.slow = 0;
  bool slow = false;
  for (int s1 = 0; s1 < b1; s1 += 2)
    for (int s2 = sym ? s1 : 0; s2 < b2; s2 += 2) {
      const bool diag = sym && s1 == s2;
      const int t1 = min(2, b1 - s1), t2 = min(2, b2 - s2);
      const int njobs = diag ? t1 : t1 + t2, ntask = diag ? t1 * (t1 + 1) / 2 : t1 * t2;
      const int split = ntask <= 2 ? 2 : 1;            // warps per pair block
      const int task = vw / split;
      const bool mine = warp >= 4 && task < ntask;
      const int c1 = diag ? (task == 2 ? 1 : 0) : task % t1, c2 = diag ? (task ? 1 : 0) : task / t1;
      const int xb = c1, yb = diag ? c2 : t1 + c2;   // operand blocks in the buffers
      const bool packed = n2 - 8 * (s2 + c2) <= 4;
      cplx acc[2] = {mkc(0.0, 0.0), mkc(0.0, 0.0)};   // packed: .x alone
      __syncthreads();   // the buffers and sums of the tile before are free
      if (warp < 4)
        hole_cut<F32>(sh, d, Yp, slow, warp < njobs, diag || warp < t1, 8 * (diag || warp < t1 ? s1 + warp : s2 + warp - t1),
                      nfib, g0, g1);
      else
        hole_mul(sh, acc, mine, packed, xb, yb, split, vw & 1, g0, g1);
      // sums: a pair block's 8 x 8, its two halves of the fibres apart where it is split
      if (mine) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (packed) {
            double* o = reinterpret_cast<double*>(&sh.sum[vw][g + 8 * (2 * (q & 1) + i)]) + (q >> 1);
            *o = acc[i].x;
          } else {
            sh.sum[vw][g + 8 * (2 * q + i)] = acc[i];
          }
        }
      }
      __syncthreads();
      for (int e = tid; e < ntask * 64; e += 64 * HOLE_WARPS) {
        const int tk = e >> 6, pr = e & 63;
        const int a1 = diag ? (tk == 2 ? 1 : 0) : tk % t1, a2 = diag ? (tk ? 1 : 0) : tk / t1;
        const int j1 = 8 * (s1 + a1) + (pr & 7), j2 = 8 * (s2 + a2) + (pr >> 3);
        if (j1 >= n1 || j2 >= n2) continue;
        cplx v = sh.sum[split * tk][pr];
        if (split == 2) v = cadd(v, sh.sum[2 * tk + 1][pr]);
        out[j1 + n1 * j2] = v;
        if (sym && s1 + a1 != s2 + a2) out[j2 + n1 * j1] = cconj(v);
      }
    }
  if (slow) sh.slow = 1;
  __syncthreads();
  if (sh.slow) hole_block_fp64(d, Yp, b, 16u * g0, min(16u * g1, nfib));
}

// The block that finishes last adds the descriptor's partials into the first, in
// block order, and resets the counter for the next launch.
template <int W>
__device__ __forceinline__ void hole_sum_blocks(const HoleDesc& d) {
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
  while (2 * sub * npairs <= 32 * W && 2 * sub <= min(nblk, 32)) sub *= 2;
  for (int w0 = 0; w0 < npairs * sub; w0 += 32 * W) {
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
// Descriptors with n1, n2 <= 8 and the wider ones go by launches of their own: each
// form has the registers and the shared memory it needs.
template <bool F32>
__global__ void __launch_bounds__(32 * HOLE_WARPS, 3)
    hole_fx_kernel(const HoleDesc* __restrict__ descs, int ndesc, long long nblocks, const cplx* ybase) {
  for (long long bb = blockIdx.x; bb < nblocks; bb += gridDim.x) {
    const HoleDesc& d = descs[warp_find_desc(descs, ndesc, bb)];
    if (bb != blockIdx.x) __syncthreads();   // the shared sums are rewritten
    hole_fx_block<F32>(d, (int)(bb - d.block_start), ybase);
    hole_sum_blocks<HOLE_WARPS>(d);
  }
}
template <bool F32>
__global__ void __launch_bounds__(64 * HOLE_WARPS, 2)
    hole_wide_kernel(const HoleDesc* __restrict__ descs, int ndesc, long long first, long long nblocks, const cplx* ybase,
                     int nsm) {
  for (long long bb = blockIdx.x; bb < nblocks; bb += gridDim.x) {
    const HoleDesc& d = descs[warp_find_desc(descs, ndesc, first + bb)];
    if (bb != blockIdx.x) __syncthreads();
    hole_wide_block<F32>(d, (int)(first + bb - d.block_start), ybase, nsm);
    hole_sum_blocks<2 * HOLE_WARPS>(d);
  }
}

template <bool F32>
static void hole_fx_go(const HoleLaunch& b, int persist, cudaStream_t st, const cplx* ybase) {
  auto grid = [&](long long n) { return (unsigned)(persist > 0 ? std::min<long long>(n, persist) : n); };
  const long long wide = b.nblocks - b.narrow_blocks;
  if (b.narrow_blocks > 0)
    hole_fx_kernel<F32><<<grid(b.narrow_blocks), 32 * HOLE_WARPS, sizeof(cplx) * 64 * HOLE_WARPS, st>>>(
        b.d, b.nnarrow, b.narrow_blocks, ybase);
  if (wide > 0)
    hole_wide_kernel<F32><<<grid(wide), 64 * HOLE_WARPS, sizeof(HoleWide), st>>>(
        b.d + b.nnarrow, b.ndesc - b.nnarrow, b.narrow_blocks, wide, ybase, sm_count());
}

void launch_hole_fx(const HoleLaunch& b, cudaStream_t st, int persist, const cplx* ybase) {
  if (b.f32) hole_fx_go<true>(b, persist, st, ybase);
  else hole_fx_go<false>(b, persist, st, ybase);
}

cudaError_t configure_fx() {
  cudaError_t e = allow_smem(prod_fx_kernel<8>, prod_smem<8>());   // the others' is below 48 KB
  static_assert(prod_smem<6>() <= 48 * 1024, "needs the opt-in");
  if (e == cudaSuccess) e = allow_smem(hole_wide_kernel<false>, sizeof(HoleWide));
  if (e == cudaSuccess) e = allow_smem(hole_wide_kernel<true>, sizeof(HoleWide));
  return e;
}
