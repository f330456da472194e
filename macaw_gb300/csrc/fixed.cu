// Mode products and single-hole contractions of FP64 accuracy as digit products on the
// tensor cores (fixed.cuh) for sm_103a: precision 0, and the FP64-accurate products and
// contractions of the mixed modes.
#include <algorithm>

#include "kernels.cuh"
#include "fixed.cuh"

// ---------------------------------------------------------------------------
// Batched mode product (Mult_HeM_MatV / Mult_GM_MatV, gmctdh_objects.f90:1407-1468)
// A warp owns 16 fibres (l, :, r) (the rows of the MMA), the columns are the (re, im)
// of four outputs j'; a lane loads elements j = q, q + 4, .. of fibres g and g + 8 and
// receives outputs q, q + 4, .. of the same fibres, so neither side passes through
// shared memory.  A fibre shares one exponent, a matrix row another, after the input
// index is scaled (fx_column_scale); sums that stay small are computed again in FP64.
// Bound by instruction issue: cutting digits and joining sums (about 50 instructions per
// complex element), not by the MMAs.
// ---------------------------------------------------------------------------

#define PROD_THREADS 128
// resident CTAs per SM the register budget is set for
template <int NJ>
constexpr int prod_ctas() {
  return NJ <= 2 ? 4 : (NJ <= 4 ? 3 : 2);
}
// NJ: groups of four j.  The CTAs share the batch's fibres evenly, each walking a
// contiguous run (its matrix digits are cut once per descriptor, the next fibres'
// loads are in flight during the products).  split: few fibres in the batch -- a unit
// is 16 fibres and the four warps share the output groups, else 64 fibres.
template <int NJ>
__global__ void __launch_bounds__(PROD_THREADS, prod_ctas<NJ>())
    prod_fx_kernel(const ProdDesc* __restrict__ descs, int ndesc, long long nblocks, int split) {
  constexpr int NS = FX_NS;
  constexpr int NK = (NJ + 1) / 2;            // k steps of 8 j; the last one of 4 for odd NJ
  constexpr bool BIG = NJ > 4;                // |D| may pass 2^22
  extern __shared__ uint2 Ws[];               // [NJ out groups][NK][NS][32]
  __shared__ unsigned rowexp[4 * NJ];         // exponent words of the matrix rows
  __shared__ unsigned colmag[4 * NJ];         // sizes of the input columns
  __shared__ int s_bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int upb = split ? 8 : 2, ufib = split ? 16 : 64;   // units per 128-fibre block, fibres per unit
  const long long nunits = upb * nblocks;
  long long u0 = nunits * blockIdx.x / gridDim.x;
  const long long uend = nunits * (blockIdx.x + 1) / gridDim.x;
  int di = warp_find_desc(descs, ndesc, u0 / upb);
  for (; u0 < uend; ++di) {
    const ProdDesc& d = descs[di];
    const int nin = d.nin, nout = d.nout, sh = fx_headroom(nin);
    const float pw = fx_pow2(sh);
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
    fx_column_sizes(d, colmag);
    __syncthreads();
    unsigned scale[NJ];
    bool scaled;
    {
      const unsigned b = fx_column_scale(colmag, nin);
      scaled = __any_sync(0xffffffffu, b);
#pragma unroll
      for (int k = 0; k < NJ; ++k) scale[k] = __shfl_sync(0xffffffffu, b, 4 * k + q);
    }
    for (int t = warp; t < nt; t += 4) {
      cplx mv[NJ];
      unsigned mag = 0;
      const int jo = 4 * t + (g >> 1);
#pragma unroll
      for (int k = 0; k < NJ; ++k) {
        const int j = 4 * k + q;
        mv[k] = mkc(0.0, 0.0);
        if (jo < nout && j < nin) mv[k] = d.conjT ? cconj(d.M[j + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * j];
        mag = max(mag, fx_scaled_down(fx_mag(mv[k]), scale[k]));
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
        const int k1 = 2 * kk + 1 < NJ ? 2 * kk + 1 : 0;
        const unsigned e0 = eb + scale[2 * kk], e1 = eb + scale[k1];
        fx_digits(mv[2 * kk].x, mv[2 * kk].y, e0, e0, s0);
        if (2 * kk + 1 < NJ) fx_digits(mv[k1].x, mv[k1].y, e1, e1, s1);
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
      unsigned limit[2];
      unsigned A[NK][NS][4];   // digits: (fibre g, j), (fibre g + 8, j), (g, j + 4), (g + 8, j + 4)
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        unsigned mag = 0u;
        if (scaled) {
#pragma unroll
          for (int k = 0; k < NJ; ++k) x[f][k] = fx_scale_up(x[f][k], scale[k]);
        }
#pragma unroll
        for (int k = 0; k < NJ; ++k) mag = max(mag, fx_mag(x[f][k]));
        mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 1));
        mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 2));
        bad = bad || !fx_ok(mag);
        limit[f] = mag ? fx_small_limit(sh) : 0u;
        const unsigned eb = fx_ebits(mag);
        ef[f] = fx_exp(eb, 0u, 44 + sh);
#pragma unroll
        for (int k = 0; k < NJ; ++k) {
          unsigned s[NS];
          fx_digits(x[f][k].x, x[f][k].y, eb, eb, s);
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
      unsigned small[2] = {0u, 0u};   // outputs left to FP64
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
          cplx kept[2];
          if (4 * t + q < nout) {
#pragma unroll
            for (int f = 0; f < 2; ++f) {
              const unsigned es = em + ef[f];
              const long long re = BIG ? fx_join_wide(c, 2 * f, pw) : fx_join(c, 2 * f, pw);
              const long long im = BIG ? fx_join_wide(c, 2 * f + 1, pw) : fx_join(c, 2 * f + 1, pw);
              cplx v = mkc(fx_double(re, es), fx_double(im, es));
              if (!plain) {
                v = cmul(d.alpha, v);
                if (d.accumulate && act[f]) v = cadd(v, y[f][t * s4]);
              }
              const bool sm = fx_small(re, im, limit[f]);
              if (sm) small[f] |= 1u << t;
              if (!sm && act[f]) y[f][t * s4] = v;
              kept[f] = v;
            }
          }
          if (__any_sync(0xffffffffu, (small[0] | small[1]) >> t & 1)) {   // one more MMA: T of these outputs
            float ct[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kk = 0; kk < NK; ++kk) {
              const uint2 w0 = Ws[(t * NK + kk) * NS * 32 + lane], w1 = Ws[((t * NK + kk) * NS + 1) * 32 + lane];
              unsigned a[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) a[k] = 2 * kk + 1 < NJ || k < 2 ? fx_lead(A[kk][0][k], A[kk][1][k]) : 0u;
              fx_mma16(ct, a, fx_lead(w0.x, w1.x), fx_lead(w0.y, w1.y), false);
            }
#pragma unroll
            for (int f = 0; f < 2; ++f)
              if ((small[f] >> t & 1) && ct[2 * f] + ct[2 * f + 1] >= FX_LOW) {
                small[f] ^= 1u << t;
                if (act[f]) y[f][t * s4] = kept[f];
              }
          }
        }
      }
      if (small[0]) prod_outputs_fp64(d, pp, small[0], q, 4);
      if (small[1]) prod_outputs_fp64(d, pp + 8, small[1], q, 4);
    }
    u0 = dend;
  }
}

template <int NJ>
constexpr int prod_smem() {
  return NJ * ((NJ + 1) / 2) * FX_NS * 32 * (int)sizeof(uint2);
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
// take 229 us against 271, of 248,832 fibres of 12 2,560 against 3,230; just above the
// line, with 6 to 8 SPFs, 22 against 27.  Below it a batch of 700 tiles of 5 to 9 took
// 19 against 17 (measured before either kernel formed T).
void launch_prod_fx(const ProdDesc* d, int nd, long long nblocks, int maxn, bool plain, int* status, cudaStream_t st,
                    int persist) {
  if (plain && persist <= 0 && tc_enabled() && maxn > 4 && maxn <= 16 && nblocks >= (maxn <= 8 ? 8 : 4) * (long long)sm_count()) {
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
// warp takes a quarter of it in groups of 16 fibres: the MMA's rows are (re, im) of eight
// X columns, its columns the re, then the im of eight Y columns, its inner dimension the
// fibres; lanes load what they hold, nothing is staged.  A column has one exponent per
// window of at most HOLE_FLUSH groups, from the window's first group; elements above it
// end the window.  A window's sums go to FP64, exactly but for the dropped digits.  One more
// MMA sums |x||y| of the leading digits: pairs where that is below 2^-6 .. 2^-8 of the
// product of the columns' largest elements (columns graded in opposite directions) are
// summed again in FP64.  On states of the models here that is none to one window in a
// hundred, and the windows of 128 neighbouring fibres are what keeps it so (interleaved
// over the warps, one in ten).  The last block of a descriptor to finish adds the blocks'
// partials in block order into the first.  42 contractions of 32,768 fibres of 8: 148 us,
// of which 14 are for windows and |x||y|; bound by cutting operands (ALU).
// ---------------------------------------------------------------------------
#define HOLE_FLUSH 8     // groups of 16 fibres between flushes: 128 x 8 x 2^14 = 2^24
#define HOLE_WARPS 4     // per block; twice as many where n1 or n2 is above eight
#define HOLE_LOW 131072.f   // 2^17 where the columns' exponents allow products of up to 2^28
// A window's exponent for a column of largest magnitude m in its first group: two binary
// orders above, so that it holds for most windows (one flush per window and a bit on the
// models' states; from the groups seen before, up to a quarter of the windows came out
// small against columns that had fallen meanwhile).  HOLE_ZERO: nothing but zeros.
#define HOLE_ZERO ((unsigned)FX_EMIN << 20)
__device__ __forceinline__ unsigned hole_exponent(unsigned m) {
  return m ? max((m & FX_EBITS) + (2u << 20), (unsigned)(FX_EMIN + 1) << 20) : HOLE_ZERO;
}
__device__ __forceinline__ bool hole_outgrown(unsigned e, unsigned m) {
  return m >= e + (1u << 20) || (e == HOLE_ZERO && m);
}

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
// exponent range (fibres p0 .. p1): a pair per warp, its lanes over the fibres.  With every
// block of the 42 contractions of 32,768 fibres of 8 here: 1,454 us against 148.
static __device__ __noinline__ void hole_block_fp64(const HoleDesc& d, const cplx* Y, int b, unsigned p0, unsigned p1) {
  const long long L = d.L;
  const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  for (int pr = threadIdx.x >> 5; pr < d.n1 * d.n2; pr += nwarp) {
    const int j1 = pr % d.n1, j2 = pr / d.n1;
    cplx acc = mkc(0, 0);
    for (long long p = p0 + lane; p < p1; p += 32) {
      const long long r = p / L, l = p - r * L;
      cfma_conj(acc, load_c(d.X, l + L * (j1 + (long long)d.n1 * r), d.xfmt),
                load_c(Y, l + L * (j2 + (long long)d.n2 * r), d.yfmt));
    }
    for (int o = 16; o > 0; o >>= 1)
      acc = cadd(acc, mkc(__shfl_xor_sync(0xffffffffu, acc.x, o), __shfl_xor_sync(0xffffffffu, acc.y, o)));
    if (lane == 0) d.partial[(long long)b * d.n1 * d.n2 + pr] = acc;
  }
}

// A pair of a window in FP64, by the whole warp: groups first, first + step, .. below last,
// fibres below nfib.
static __device__ __noinline__ cplx hole_pair_fp64(const HoleDesc& d, const cplx* Y, unsigned first, unsigned last,
                                                   unsigned step, unsigned nfib, int j1, int j2) {
  const long long L = d.L;
  const unsigned n = 16 * ((last - first + step - 1) / step);
  cplx v = mkc(0, 0);
  for (unsigned f = threadIdx.x & 31; f < n; f += 32) {
    const unsigned p = 16 * (first + step * (f >> 4)) + (f & 15);
    if (p >= nfib) break;
    const long long r = p / L, l = p - r * L;
    cfma_conj(v, load_c(d.X, l + L * (j1 + (long long)d.n1 * r), d.xfmt), load_c(Y, l + L * (j2 + (long long)d.n2 * r), d.yfmt));
  }
  for (int o = 16; o > 0; o >>= 1)
    v = cadd(v, mkc(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)));
  return v;
}

// F32: operands may be complex FP32
// What a sum may still be off by: `credit` is T - HOLE_LOW B, T = sum |x||y| so far and B the
// number of windows taken from digits, each in units of the windows' own 2^(ex + ey).  A
// window of which T adds t is taken if that leaves the credit positive.
__device__ __forceinline__ bool hole_credit(float& credit, float t) {
  const bool take = credit + t >= HOLE_LOW;
  credit += take ? t - HOLE_LOW : t;
  return take;
}
// ... in the units of new exponents
__device__ __forceinline__ float hole_rescale(unsigned was, unsigned now) {
  const int e = (int)(was - now) >> 20;
  return __uint_as_float((unsigned)(min(max(e, -126), 120) + 127) << 23);
}

// The windows of a warp's pairs that are left to FP64: noted while the sums are in
// registers, done at the end by all warps of the block, added in their order.
#define HOLE_LATE 128
struct HoleLate {
  int n;
  unsigned first[HOLE_LATE], last[HOLE_LATE];
  unsigned char pair[HOLE_LATE];   // 2 lane + column
};
__device__ __forceinline__ void hole_note(HoleLate& t, bool low, int i, unsigned first, unsigned last) {
  const unsigned who = __ballot_sync(0xffffffffu, low), lane = threadIdx.x & 31;
  if (!who) return;
  const int k = t.n + __popc(who & ((1u << lane) - 1u));
  __syncwarp();
  if (low && k < HOLE_LATE) {
    t.first[k] = first;
    t.last[k] = last;
    t.pair[k] = (unsigned char)(2 * lane + i);
  }
  if (lane == 0) t.n += __popc(who);
  __syncwarp();
}

struct HoleNarrow {
  union {
    cplx raw[HOLE_WARPS][2][8][32];   // operands in flight: [warp][slot][X's four, then Y's four fibres][lane]
    struct {
      cplx red[HOLE_WARPS][64];
      cplx val[HOLE_WARPS][HOLE_LATE];
    };
  };
  HoleLate late[HOLE_WARPS];
};
__device__ __forceinline__ void hole_copy(unsigned dst, const cplx* P, long long e, int fmt, bool in) {
  if (fmt)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(reinterpret_cast<const float2*>(P) + (in ? e : 0)), "r"(in ? 8 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(P + (in ? e : 0)), "r"(in ? 16 : 0) : "memory");
}

template <bool F32>
__device__ __forceinline__ void hole_fx_block(const HoleDesc& d, int b, const cplx* ybase) {
  constexpr int NS = FX_NS, W = HOLE_WARPS;
  extern __shared__ __align__(16) unsigned char hole_sm[];
  HoleNarrow& sh = *reinterpret_cast<HoleNarrow*>(hole_sm);
  __shared__ int s_slow;
  const cplx* Yp = d.Y ? d.Y : ybase + d.yoff;
  const int n1 = d.n1, n2 = d.n2, npairs = n1 * n2;
  if (npairs == 1 && d.Y && d.L * d.R >= 32 * W) {
    dot_block(d, b, sh.red[0]);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int xfmt = F32 ? d.xfmt : 0, yfmt = F32 ? d.yfmt : 0;
  // X = Y (density matrices, SPF overlaps): the digits serve both operands
  const bool same = d.X == d.Y && n1 == n2 && d.xfmt == d.yfmt;
  const unsigned L = (unsigned)d.L, nfib = (unsigned)(d.L * d.R);
  const unsigned ngrp = (nfib + 15) / 16;
  const unsigned b0 = (unsigned)((unsigned long long)ngrp * b / d.nblk);
  const unsigned b1 = (unsigned)((unsigned long long)ngrp * (b + 1) / d.nblk);
  const unsigned g0 = b0 + (b1 - b0) * warp / W, g1 = b0 + (b1 - b0) * (warp + 1) / W;   // the warp's groups
  const unsigned dl = 16u % L, dr = 16u / L;
  if (tid == 0) s_slow = 0;
  __syncthreads();
  bool slow = false;
  // the lane's columns g of X and Y, its fibres 2 q, 2 q + 1, 2 q + 8, 2 q + 9 of a group:
  // copied by the lane for itself, two groups ahead
  unsigned p = 16u * g0 + 2 * q, l[2], r[2];   // of fibres 2 q, 2 q + 8
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    r[h] = (p + 8 * h) / L;
    l[h] = p + 8 * h - L * r[h];
  }
  const unsigned raw0 = (unsigned)__cvta_generic_to_shared(&sh.raw[warp][0][0][lane]);
  constexpr unsigned SLOT = sizeof(sh.raw[0][0]), FIB = sizeof(sh.raw[0][0][0]);
  unsigned ahead = g0;
  auto fetch = [&](unsigned slot) {
    if (ahead < g1) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool wrap = l[h] + 1 == L;
        const unsigned l1 = wrap ? 0u : l[h] + 1, r1 = wrap ? r[h] + 1 : r[h];
        const bool i0 = p + 8 * h < nfib, i1 = p + 8 * h + 1 < nfib;
        const unsigned dst = raw0 + slot * SLOT + 2 * h * FIB;
        hole_copy(dst, d.X, l[h] + (long long)L * (g + (long long)n1 * r[h]), xfmt, i0 && g < n1);
        hole_copy(dst + FIB, d.X, l1 + (long long)L * (g + (long long)n1 * r1), xfmt, i1 && g < n1);
        if (!same) {
          hole_copy(dst + 4 * FIB, Yp, l[h] + (long long)L * (g + (long long)n2 * r[h]), yfmt, i0 && g < n2);
          hole_copy(dst + 5 * FIB, Yp, l1 + (long long)L * (g + (long long)n2 * r1), yfmt, i1 && g < n2);
        }
        l[h] += dl;
        r[h] += dr;
        if (l[h] >= L) { l[h] -= L; r[h] += 1; }
      }
      p += 16;
      ++ahead;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float cr[8][4], ci[8][4], ct[4];   // sums with Yr and Yi: rows Xr (0, 1), Xi (2, 3); |x||y| alike
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ct[i] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) cr[k][i] = ci[k][i] = 0.f;
    }
  };
  clear();
  cplx acc[2] = {mkc(0.0, 0.0), mkc(0.0, 0.0)};
  float credit[2] = {0.f, 0.f};
  constexpr unsigned emax = (unsigned)(FX_EMAX + 1) << 20;
  unsigned ex = HOLE_ZERO, ey = HOLE_ZERO, gw = g0;   // exponents, the window's first group
  auto flush = [&](unsigned gend) {
    // conj(x) y = (Xr Yr + Xi Yi) + i (Xr Yi - Xi Yr) of columns 2 q, 2 q + 1
    const unsigned ec = same ? ex : ey;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned e2 = __shfl_sync(0xffffffffu, ec, 8 * q + 4 * i), es = fx_exp(ex, e2, 24);
      long long hi, lo;
      cplx v;
      fx_join_pair<false>(cr, i, ci, 2 + i, hi, lo);
      v.x = fx_double_pair(hi, lo, es);
      fx_join_pair<true>(ci, i, cr, 2 + i, hi, lo);
      v.y = fx_double_pair(hi, lo, es);
      const bool low = ex != HOLE_ZERO && e2 != HOLE_ZERO && !hole_credit(credit[i], ct[i] + ct[2 + i]);
      hole_note(sh.late[warp], low, i, gw, gend);
      if (!low) acc[i] = cadd(acc[i], v);
    }
    clear();
  };
  if (lane == 0) sh.late[warp].n = 0;
  __syncwarp();
  fetch(0);
  fetch(1);
  unsigned slot = 0;
  for (unsigned gr = g0; gr < g1; ++gr, slot ^= 1) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const cplx* px = &sh.raw[warp][slot][0][lane];
    const cplx* py = px + 4 * 32;
    auto xel = [&](int f) { return load_c(px + 32 * f, 0, xfmt); };
    auto yel = [&](int f) { return load_c(py + 32 * f, 0, yfmt); };
    unsigned mx = max(max(fx_mag(xel(0)), fx_mag(xel(1))), max(fx_mag(xel(2)), fx_mag(xel(3))));
    unsigned my = same ? 0u : max(max(fx_mag(yel(0)), fx_mag(yel(1))), max(fx_mag(yel(2)), fx_mag(yel(3))));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    my = max(my, __shfl_xor_sync(0xffffffffu, my, 1));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    my = max(my, __shfl_xor_sync(0xffffffffu, my, 2));
    slow = slow || mx >= emax || my >= emax;
    const bool grow = hole_outgrown(ex, mx) || hole_outgrown(ey, my);
    if (__any_sync(0xffffffffu, grow) || gr - gw == HOLE_FLUSH) {
      if (gr != gw) flush(gr);
      const unsigned wasx = ex, was2 = same ? ex : ey;
      ex = hole_exponent(mx);
      ey = hole_exponent(my);
      const unsigned now2 = same ? ex : ey;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        credit[i] *= hole_rescale(wasx + __shfl_sync(0xffffffffu, was2, 8 * q + 4 * i),
                                  ex + __shfl_sync(0xffffffffu, now2, 8 * q + 4 * i));
      gw = gr;
    }
    unsigned A[NS][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unsigned s[NS];
      const cplx x0 = xel(2 * h), x1 = xel(2 * h + 1);
      fx_digits(x0.x, x1.x, ex, ex, s);
#pragma unroll
      for (int k = 0; k < NS; ++k) A[k][2 * h] = s[k];
      fx_digits(x0.y, x1.y, ex, ex, s);
#pragma unroll
      for (int k = 0; k < NS; ++k) A[k][2 * h + 1] = s[k];
    }
    // the re, then the im of Y: one set of digits at a time
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      unsigned B[NS][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (same) {
#pragma unroll
          for (int k = 0; k < NS; ++k) B[k][h] = A[k][2 * h + part];
        } else {
          unsigned s[NS];
          const cplx y0 = yel(2 * h), y1 = yel(2 * h + 1);
          if (part == 0) fx_digits(y0.x, y1.x, ey, ey, s);
          else fx_digits(y0.y, y1.y, ey, ey, s);
#pragma unroll
          for (int k = 0; k < NS; ++k) B[k][h] = s[k];
        }
      }
      if (part == 1) fetch(slot);   // the slot is read
      {
        unsigned t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = fx_lead(A[0][i], A[1][i]);
        fx_mma16(ct, t, fx_lead(B[0][0], B[1][0]), fx_lead(B[0][1], B[1][1]), false);
      }
#pragma unroll
      for (int i = 0; i < NS; ++i)
#pragma unroll
        for (int j = 0; j + i < NS; ++j) fx_mma16(part ? ci[i + j] : cr[i + j], A[i], B[j][0], B[j][1], false);
    }
  }
  if (g0 < g1) flush(g1);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (slow || sh.late[warp].n > HOLE_LATE) s_slow = 1;
  __syncthreads();   // every operand is cut: the sums take their place
  for (int w = 0; w < W; ++w)
    for (int k = warp; k < min(sh.late[w].n, HOLE_LATE); k += W) {
      const HoleLate& t = sh.late[w];
      const int src = t.pair[k] >> 1;
      const cplx o = hole_pair_fp64(d, Yp, t.first[k], t.last[k], 1, nfib, src >> 2, 2 * (src & 3) + (t.pair[k] & 1));
      if (lane == 0) sh.val[w][k] = o;
    }
  __syncthreads();
  for (int k = 0; k < min(sh.late[warp].n, HOLE_LATE); ++k)
    if (sh.late[warp].pair[k] >> 1 == lane) {
      if (sh.late[warp].pair[k] & 1) acc[1] = cadd(acc[1], sh.val[warp][k]);
      else acc[0] = cadd(acc[0], sh.val[warp][k]);
    }
  // (j1, j2) = (g, 2 q), (g, 2 q + 1)
  sh.red[warp][g + 8 * (2 * q)] = acc[0];
  sh.red[warp][g + 8 * (2 * q + 1)] = acc[1];
  __syncthreads();
  if (s_slow) {
    hole_block_fp64(d, Yp, b, 16u * b0, min(16u * b1, nfib));
    return;
  }
  cplx* out = d.partial + (long long)b * npairs;
  for (int pr = tid; pr < npairs; pr += 32 * W) {
    const int e = pr % n1 + 8 * (pr / n1);
    cplx v = sh.red[0][e];
    for (int k = 1; k < W; ++k) v = cadd(v, sh.red[k][e]);
    out[pr] = v;
  }
}

// The same for n1 or n2 above eight.  Tiles of two by two column blocks: each operand
// block of 32 fibres is cut once, by one warp, into shared memory in the order the MMAs
// read it (an uint4 per lane, digit and group of 16 fibres: re, im of fibres 2 q, 2 q + 1,
// then of 2 q + 8, 2 q + 9), and every warp takes a pair block of the tile.  Where every
// pair block cut its own operands, cutting bound the kernel (ALU 52 %, tensor pipe 36 %).
// 42 contractions of 12 SPFs (8,957,952 coefficients): 3,040 us, of which 760 are for the
// exponents of windows and the sums |x||y|.
// A column block of at most four columns puts re and im side by side into one MMA.
// Warps 0-3 cut the next stage while warps 4-7 multiply this one: with every warp doing
// both in turn the phases of a block did not overlap.
// Windows, exponents and the FP64 of small pairs as above; a new window at every
// HOLEW_FLUSH-th stage.
#define HOLEW_GRP 2      // groups of 16 fibres per stage
#define HOLEW_FLUSH (HOLE_FLUSH / HOLEW_GRP)
#define HOLEW_SLOTS 2    // stages of operands in flight
struct HoleWide {
  uint4 dig[2][4][HOLEW_GRP][FX_NS][32];     // [buffer][operand block][group][digit][lane]
  cplx raw[HOLEW_SLOTS][4][4 * HOLEW_GRP][32];  // operands: [slot][block][fibre of the lane][lane]
  cplx acc[4][2][32];                        // a multiplier's sums: [warp][column][lane] (packed: .x alone)
  float credit[4][2][32];
  HoleLate late[4];
  unsigned ex[4][4][8];                      // the columns' exponents in four successive stages
  int grow[2][4];
  int slow;
};
static_assert(2 * (sizeof(HoleWide) + 1024 + 64) <= 228 * 1024, "two CTAs per SM");
// both roles pass the same barriers: one before the first stage, one after each
__device__ __forceinline__ void hole_stage_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(64 * HOLE_WARPS) : "memory");
}
template <bool F32>
__device__ __forceinline__ void hole_cut(HoleWide& sh, const HoleDesc& d, const cplx* Yp, bool& slow, bool cut, bool isx,
                                         int j0, unsigned nfib, unsigned g0, unsigned g1) {
  constexpr int NS = FX_NS, NP = 4 * HOLEW_GRP;   // fibres per lane and stage
  constexpr unsigned emax = (unsigned)(FX_EMAX + 1) << 20;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const unsigned L = (unsigned)d.L, dl = (16u * HOLEW_GRP) % L, dr = (16u * HOLEW_GRP) / L;
  const cplx* P = isx ? d.X : Yp;
  const int np = isx ? d.n1 : d.n2, j = j0 + g;
  const int fmt = F32 ? (isx ? d.xfmt : d.yfmt) : 0;
  unsigned grp = g0, ec = HOLE_ZERO, l[NP / 2], r[NP / 2];   // fibres 2 q (+ 8) of each group
#pragma unroll
  for (int h = 0; h < NP / 2; ++h) {
    const unsigned p = 16 * g0 + 8 * h + 2 * q;
    r[h] = p / L;
    l[h] = p - L * r[h];
  }
  const unsigned raw0 = (unsigned)__cvta_generic_to_shared(&sh.raw[0][warp][0][lane]);
  constexpr unsigned slot_bytes = sizeof(sh.raw[0]), point_bytes = sizeof(sh.raw[0][0][0]);
  auto copy = [&](unsigned dst, unsigned ll, unsigned rr, bool in) {
    hole_copy(dst, P, ll + (long long)L * (j + (long long)np * rr), fmt, in);
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
  auto stage = [&](int buf, int st) {   // cut the oldest stage in flight, number st, into buffer buf
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
    slow = slow || m >= emax;
    const bool any = __any_sync(0xffffffffu, st % HOLEW_FLUSH == 0 || hole_outgrown(ec, m));
    if (any) ec = hole_exponent(m);
    if (lane == 0) sh.grow[buf][warp] = any;
    if (q == 0) sh.ex[st & 3][warp][g] = ec;
#pragma unroll
    for (int gg = 0; gg < HOLEW_GRP; ++gg) {
      unsigned s[4][NS];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        fx_digits(x[4 * gg + 2 * h].x, x[4 * gg + 2 * h + 1].x, ec, ec, s[2 * h]);
        fx_digits(x[4 * gg + 2 * h].y, x[4 * gg + 2 * h + 1].y, ec, ec, s[2 * h + 1]);
      }
#pragma unroll
      for (int k = 0; k < NS; ++k) sh.dig[buf][warp][gg][k][lane] = make_uint4(s[0][k], s[1][k], s[2][k], s[3][k]);
    }
  };
  for (int k = 0; k < HOLEW_SLOTS; ++k) fetch();
  if (cut) stage(0, 0);
  fetch();
  hole_stage_barrier();
  int buf = 1, st = 1;
  for (unsigned gr = g0; gr < g1; gr += HOLEW_GRP, buf ^= 1, ++st) {
    if (cut && gr + HOLEW_GRP < g1) stage(buf, st);
    fetch();
    hole_stage_barrier();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}
// The pair block (xb, yb) of the buffers.
template <bool PACKED>
__device__ __forceinline__ void hole_mul_go(HoleWide& sh, int vw, bool mine, int xb, int yb, int split, unsigned g0,
                                            unsigned g1) {
  constexpr int NS = FX_NS;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, cy = PACKED ? 2 * (q & 1) : 2 * q;
  float cr[8][4], ci[8][4], ct[4];   // sums with Yr and Yi (packed: all in cr): rows Xr (0, 1), Xi (2, 3); |x||y|
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ct[i] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) cr[k][i] = ci[k][i] = 0.f;
    }
  };
  clear();
  const int half = vw & 1;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    sh.acc[vw][i][lane] = mkc(0.0, 0.0);
    sh.credit[vw][i][lane] = 0.f;
  }
  if (lane == 0) sh.late[vw].n = 0;
  __syncwarp();
  unsigned gw = g0;
  auto flush = [&](unsigned gend, const unsigned (*ex)[8]) {   // ex: of the window's stages
    const unsigned e1 = ex[xb][g], first = gw + (split == 2 ? half : 0);   // of the groups of this warp's half
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned e2 = ex[yb][cy + i], es = fx_exp(e1, e2, 24);
      long long hi, lo;
      float t = ct[i] + ct[2 + i];
      cplx v;
      if (PACKED) {
        // conj(x) y of a column: re = Xr Yr + Xi Yi in lanes q < 2, im = Xr Yi - Xi Yr in q + 2
        float o[8][4];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          o[k][0] = __shfl_xor_sync(0xffffffffu, cr[k][2 + i], 2);
          if (q >= 2) o[k][0] = -o[k][0];
        }
        fx_join_pair<false>(cr, i, o, 0, hi, lo);
        v = mkc(fx_double_pair(hi, lo, es), 0.0);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
      } else {
        fx_join_pair<false>(cr, i, ci, 2 + i, hi, lo);
        v.x = fx_double_pair(hi, lo, es);
        fx_join_pair<true>(ci, i, cr, 2 + i, hi, lo);
        v.y = fx_double_pair(hi, lo, es);
      }
      const bool low = first < gend && e1 != HOLE_ZERO && e2 != HOLE_ZERO && !hole_credit(sh.credit[vw][i][lane], t);
      hole_note(sh.late[vw], low && (!PACKED || q < 2), i, first, gend);   // packed: its im is two lanes on
      cplx& a = sh.acc[vw][i][lane];
      if (!low) a = cadd(a, v);
    }
    clear();
  };
  hole_stage_barrier();
  int st = 0;
  for (unsigned gr = g0; gr < g1; gr += HOLEW_GRP, ++st) {
    const int buf = st & 1;
    if (mine) {
      if (sh.grow[buf][xb] || sh.grow[buf][yb]) {   // a new window, every HOLEW_FLUSH stages at least
        const unsigned(*was)[8] = sh.ex[(st - 1) & 3], (*now)[8] = sh.ex[st & 3];
        if (gr != g0) {
          flush(gr, was);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            sh.credit[vw][i][lane] *= hole_rescale(was[xb][g] + was[yb][cy + i], now[xb][g] + now[yb][cy + i]);
        }
        gw = gr;
      }
#pragma unroll 1
      for (int gg = split == 2 ? half : 0; gg < HOLEW_GRP; gg += split) {
        const uint4* xd = &sh.dig[buf][xb][gg][0][lane];
        // packed: columns g & 3, re for g < 4, im above
        const uint4* yd = &sh.dig[buf][yb][gg][0][PACKED ? lane & 15 : lane];
        unsigned A[NS][4];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
          const uint4 v = xd[32 * k];
          A[k][0] = v.x;
          A[k][1] = v.y;
          A[k][2] = v.z;
          A[k][3] = v.w;
        }
        {   // |x||y| of the leading digits
          unsigned t[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = fx_lead(A[0][i], A[1][i]);
          const uint4 u = yd[0], v = yd[32];
          if (PACKED)
            fx_mma16(ct, t, fx_lead(g < 4 ? u.x : u.y, g < 4 ? v.x : v.y), fx_lead(g < 4 ? u.z : u.w, g < 4 ? v.z : v.w), false);
          else
            fx_mma16(ct, t, fx_add_half2(fx_lead(u.x, v.x), fx_lead(u.y, v.y)),
                     fx_add_half2(fx_lead(u.z, v.z), fx_lead(u.w, v.w)), false);
        }
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          const uint4 v = yd[32 * j];
          const unsigned p0 = PACKED && g >= 4 ? v.y : v.x, p1 = PACKED && g >= 4 ? v.w : v.z;
#pragma unroll
          for (int i = 0; i + j < NS; ++i) {
            fx_mma16(cr[i + j], A[i], p0, p1, false);
            if (!PACKED) fx_mma16(ci[i + j], A[i], v.y, v.w, false);
          }
        }
      }
    }
    hole_stage_barrier();
  }
  if (mine && g0 < g1) flush(g1, sh.ex[(st - 1) & 3]);
}

template <bool F32>
__device__ __forceinline__ void hole_wide_block(const HoleDesc& d, int b, const cplx* ybase, int nsm) {
  extern __shared__ cplx red[];
  HoleWide& sh = *reinterpret_cast<HoleWide*>(red);
  const cplx* Yp = d.Y ? d.Y : ybase + d.yoff;
  const int n1 = d.n1, n2 = d.n2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
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
      __syncthreads();   // the buffers and sums of the tile before are free
      if (warp < 4)
        hole_cut<F32>(sh, d, Yp, slow, warp < njobs, diag || warp < t1, 8 * (diag || warp < t1 ? s1 + warp : s2 + warp - t1),
                      nfib, g0, g1);
      else if (packed)
        hole_mul_go<true>(sh, vw, mine, xb, yb, split, g0, g1);
      else
        hole_mul_go<false>(sh, vw, mine, xb, yb, split, g0, g1);
      __syncthreads();   // the operands are cut, and what is left to FP64 takes their place
      cplx(*val)[HOLE_LATE] = reinterpret_cast<cplx(*)[HOLE_LATE]>(&sh.raw[0][0][0][0]);
      for (int w = 0; w < 4; ++w) {
        const HoleLate& t = sh.late[w];
        slow = slow || t.n > HOLE_LATE;
        const int tk = w / split, a1 = diag ? (tk == 2 ? 1 : 0) : tk % t1, a2 = diag ? (tk ? 1 : 0) : tk / t1;
        for (int k = warp; k < min(t.n, HOLE_LATE); k += 2 * HOLE_WARPS) {
          const int src = t.pair[k] >> 1;
          const cplx o = hole_pair_fp64(d, Yp, t.first[k], t.last[k], split, nfib, 8 * (s1 + a1) + (src >> 2),
                                        8 * (s2 + a2) + 2 * (src & 3) + (t.pair[k] & 1));
          if (lane == 0) val[w][k] = o;
        }
      }
      __syncthreads();
      if (warp >= 4) {
        const HoleLate& t = sh.late[vw];
        for (int k = 0; k < min(t.n, HOLE_LATE); ++k) {
          const int src = t.pair[k] >> 1;
          cplx& a = sh.acc[vw][t.pair[k] & 1][lane];
          const cplx o = val[vw][k];
          if (lane == src) a = cadd(a, packed ? mkc(o.x, 0.0) : o);
          if (packed && lane == src + 2) a.x += o.y;
        }
      }
      __syncthreads();
      // the pair blocks' sums, the two halves of the fibres apart where a block is split
      for (int e = tid; e < ntask * 64; e += 64 * HOLE_WARPS) {
        const int tk = e >> 6, pr = e & 63;
        const int a1 = diag ? (tk == 2 ? 1 : 0) : tk % t1, a2 = diag ? (tk ? 1 : 0) : tk / t1;
        const int j1 = 8 * (s1 + a1) + (pr & 7), j2 = 8 * (s2 + a2) + (pr >> 3);
        if (j1 >= n1 || j2 >= n2) continue;
        const bool pk = n2 - 8 * (s2 + a2) <= 4;
        cplx v = mkc(0.0, 0.0);
        for (int h = 0; h < split; ++h) {
          const cplx* a = &sh.acc[split * tk + h][(pr >> 3) & 1][4 * (pr & 7) + (pr >> 4)];
          v = cadd(v, pk ? mkc(a[0].x, a[2].x) : a[0]);
        }
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
    hole_fx_kernel<F32><<<grid(b.narrow_blocks), 32 * HOLE_WARPS, sizeof(HoleNarrow), st>>>(
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
