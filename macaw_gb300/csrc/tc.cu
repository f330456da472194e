// Tensor-core (tcgen05, TF32 with FP32 accumulation in TMEM) kernels of the
// split-FP32 path for sm_103a.
//
// Batched mode product (Mult_HeM_MatV / Mult_GM_MatV, gmctdh_objects.f90:1407-1468)
// as a GEMM: the 128 fibres (l, :, r) of a tile are the rows, the complex
// matrix is a real 2 nin x 2 nout block [[Mr, Mi], [-Mi, Mr]] acting on the
// interleaved (re, im) columns, so D(fibre, 2 jo + c) is the real (c = 0) or
// imaginary (c = 1) part of output jo.  Every FP32 operand is split exactly into
// three TF32 numbers, x = hi + mid + lo (11 + 11 + 2 significant bits), and a
// tile takes six MMAs per K step (every part product down to 2^-22 of the
// leading one: lo*hi, mid*mid, hi*lo, mid*hi, hi*mid, hi*hi): each product is
// carried to ~2^-33, so the FP32 accumulation in TMEM is the only rounding, as
// in the FP32 CUDA-core products this replaces.
//
// Persistent CTAs of 4 warps (128 threads) walk the tiles of all descriptors
// (tile b of the batch = fibres 128 (b - block_start) ... of its descriptor, the
// CUDA-core kernel's block mapping): thread t loads fibre t of a tile (coalesced
// along l), splits it and writes the K-major operand tiles of its stage; thread
// 0 issues the MMAs into that stage's 32-column TMEM accumulator and commits
// them to the stage's mbarrier; every warp then reads its 32 TMEM lanes (= its
// 32 fibres) and stores them.  With two stages the loads of tile i run while
// the MMAs of tile i - 1 finish, and tile i - 1 is drained after them; with one
// stage a CTA drains each tile before loading the next, and twice as many CTAs
// share an SM.
#include <algorithm>
#include <mutex>
#include <stdlib.h>

#include "../../include/macaw_gb300.h"
#include "kernels.cuh"
#include "tc.cuh"
#include "fixed.cuh"

#define TC_ROWS 128
#define TC_MAXN 16          // largest nin / nout of the tensor-core mode product
#define TC_NPART 3          // hi, mid, lo

// set when a tensor-core kernel gave up waiting for its MMAs (never expected); the call
// that launched it fails by its own status word
__device__ int g_tc_timeout = 0;

// A wait ran out: results are missing, and the MMAs in flight may still write TMEM.  Wait
// once more before the caller gives TMEM back.
__device__ __forceinline__ void tc_gave_up(uint64_t* bar, uint32_t parity, int* status) {
  tc_wait(bar, parity);
  atomicExch(&g_tc_timeout, 1);
  atomicOr(status, DEVST_TC_WAIT);
}

__device__ __forceinline__ int tc_find_tile(const ProdDesc* descs, int ndesc, long long b) {
  int lo = 0, hi = ndesc - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (descs[mid].block_start <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(TC_ROWS) prod_tc_kernel(const ProdDesc* __restrict__ descs, int ndesc,
                                                          long long ntiles, int K, int N, int nstage, int* status) {
  extern __shared__ __align__(128) unsigned char tc_smem[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5;
  // stage layout: A parts (128 x K floats each), then B parts (N x K floats each)
  const uint32_t abytes = (uint32_t)TC_ROWS * K * 4, bbytes = (uint32_t)N * K * 4;
  const uint32_t sbytes = TC_NPART * (abytes + bbytes);
  const uint32_t base = tc_smem_addr(tc_smem);
  if (tid == 0) {
    tc_bar_init(&bar[0], 1);
    tc_bar_init(&bar[1], 1);
  }
  if (warp == 0) tc_alloc(&s_tmem, 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const uint32_t idesc = tc_idesc_tf32(TC_ROWS, N);
  const uint32_t sbo = (uint32_t)K * 32;
  bool ok = true;
  uint32_t late = 0;         // where a wait ran out: 2 stage + parity of the last commit
  int prev_di = -1;          // the tile loaded in the previous iteration
  long long prev_p = 0;
  int it = 0;
  for (long long tile = blockIdx.x;; tile += gridDim.x, ++it) {
    const bool have = tile < ntiles;
    const int s = (nstage == 2) ? (it & 1) : 0;
    int di = -1;
    long long p = 0;
    if (have) {
      di = tc_find_tile(descs, ndesc, tile);
      const ProdDesc& d = descs[di];
      const int nin = d.nin, nout = d.nout;
      unsigned char* sb = tc_smem + s * sbytes;
      // B(n, k): n = 2 jo + c', k = 2 ji + c; y_re = sum Mr x_re - Mi x_im, y_im = sum Mi x_re + Mr x_im
      for (int e = tid; e < N * K; e += TC_ROWS) {
        const int n = e % N, k = e / N;
        const int jo = n >> 1, ji = k >> 1;
        float v = 0.f;
        if (jo < nout && ji < nin) {
          const cplx m = d.conjT ? cconj(d.M[ji + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * ji];
          const int cout = n & 1, cin = k & 1;
          const float mr = (float)m.x, mi = (float)m.y;
          v = (cout == cin) ? mr : (cout ? mi : -mi);
        }
        float h, m_, l;
        tc_split3(v, h, m_, l);
        const uint32_t o = TC_NPART * abytes + tc_off(n, k, K);
        *reinterpret_cast<float*>(sb + o) = h;
        *reinterpret_cast<float*>(sb + o + bbytes) = m_;
        *reinterpret_cast<float*>(sb + o + 2 * bbytes) = l;
      }
      // A: fibre tid of the tile
      const long long L = d.L, nfib = d.L * d.R;
      p = (tile - d.block_start) * TC_ROWS + tid;
      const bool valid = p < nfib;
      long long l = 0, r = 0;
      if (valid) fibre_lr(p, L, nfib, l, r);
      const long long xi0 = l + L * (long long)nin * r;
      for (int k4 = 0; k4 < K; k4 += 4) {
        float x[4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int ji = (k4 >> 1) + q;
          float re = 0.f, im = 0.f;
          if (valid && ji < nin) {
            const float4 w = load_split(d.X, xi0 + L * ji, d.xfmt);
            re = w.x + w.z;
            im = w.y + w.w;
          }
          x[2 * q] = re;
          x[2 * q + 1] = im;
        }
        float4 hv, mv, lv;
        tc_split3(x[0], hv.x, mv.x, lv.x);
        tc_split3(x[1], hv.y, mv.y, lv.y);
        tc_split3(x[2], hv.z, mv.z, lv.z);
        tc_split3(x[3], hv.w, mv.w, lv.w);
        const uint32_t o = tc_off(tid, k4, K);
        *reinterpret_cast<float4*>(sb + o) = hv;
        *reinterpret_cast<float4*>(sb + o + abytes) = mv;
        *reinterpret_cast<float4*>(sb + o + 2 * abytes) = lv;
      }
    }
    tc_fence_smem();
    tc_fence_before();
    __syncthreads();
    if (have && tid == 0) {
      tc_fence_after();
      const uint32_t dt = tmem + 32u * s;
      const uint32_t sa = base + s * sbytes, sbb = sa + TC_NPART * abytes;
      // part products in increasing size: (A part, B part) = (lo, hi), (mid, mid),
      // (hi, lo), (mid, hi), (hi, mid), (hi, hi); part 0 = hi, 1 = mid, 2 = lo
      uint32_t acc = 0;
      for (int k8 = 0; k8 < K / 8; ++k8) {
        const uint32_t o = 256u * k8;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const uint32_t pa = (q == 0) ? 2u : ((q == 1 || q == 3) ? 1u : 0u);
          const uint32_t pb = (q == 2) ? 2u : ((q == 1 || q == 4) ? 1u : 0u);
          tc_mma_tf32(dt, tc_smem_desc(sa + pa * abytes + o, 128, sbo), tc_smem_desc(sbb + pb * bbytes + o, 128, sbo),
                      idesc, acc);
          acc = 1;
        }
      }
      tc_commit(&bar[s]);
    }
    // Drain: with two stages the previous tile (the other stage) while this one
    // runs, with one stage this tile.  Uniform across the CTA.
    const bool do_drain = (nstage == 2) ? (prev_di >= 0) : have;
    if (do_drain) {
      const int ps = (nstage == 2) ? ((it - 1) & 1) : 0;
      const uint32_t parity = (nstage == 2) ? ((uint32_t)((it - 1) >> 1) & 1u) : ((uint32_t)it & 1u);
      const int dd = (nstage == 2) ? prev_di : di;
      const long long dpf = (nstage == 2) ? prev_p : p;
      // every thread polls the mbarrier; the verdict is made uniform across the
      // CTA so that all threads leave the loop together if a wait ran out
      const bool w = __syncthreads_and(tc_wait(&bar[ps], parity));
      tc_fence_after();
      if (!w) {
        ok = false;
        late = nstage == 2 && have ? 2 * s + ((uint32_t)(it >> 1) & 1u) : 2 * ps + parity;
      } else {
        const ProdDesc& d = descs[dd];
        const int nout = d.nout;
        float acc[32];
        const uint32_t trow = tmem + 32u * ps + ((uint32_t)(warp * 32) << 16);
        tc_ld16(trow, acc);
        if (N > 16) tc_ld16(trow + 16, acc + 16);
        const long long L = d.L, nfib = d.L * d.R;
        if (dpf < nfib) {
          long long l, r;
          fibre_lr(dpf, L, nfib, l, r);
          cplx* y0 = d.Y + l + L * (long long)nout * r;
          float4* y0f = reinterpret_cast<float4*>(y0);
          const bool unit_alpha = (d.alpha.x == 1.0 && d.alpha.y == 0.0);
#pragma unroll
          for (int jo = 0; jo < TC_MAXN; ++jo) {
            if (jo >= nout) break;
            const float re = acc[2 * jo], im = acc[2 * jo + 1];
            if (d.yfmt == TF_F32) {
              reinterpret_cast<float2*>(d.Y)[l + L * ((long long)nout * r + jo)] = make_float2(re, im);
            } else if (d.yfmt) {
              y0f[L * jo] = make_float4(re, im, 0.f, 0.f);
            } else {
              const cplx a = mkc(f2d_exact(re), f2d_exact(im));
              cplx v = unit_alpha ? a : cmul(d.alpha, a);
              if (d.accumulate) v = cadd(v, y0[L * jo]);
              y0[L * jo] = v;
            }
          }
        }
      }
    }
    if (!have || !ok) break;
    prev_di = di;
    prev_p = p;
  }
  if (!ok && tid == 0) tc_gave_up(&bar[late >> 1], late & 1, status);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tc_dealloc(tmem, 64);
  }
}

// ---------------------------------------------------------------------------
// Mode products of FP64 accuracy as digit products (fixed.cuh) with tcgen05 (factors of
// one, nothing accumulated: ProdBatch::plain).  A tile is 128 fibres, one per thread and
// MMA row; the thread cuts its fibre into eight FP16 digits of one exponent, digit i of
// all fibres being operand A_i (128 x 2 nin).  The matrix's digits lie side by side as
// columns, B = [B_0 B_1 .. B_7] (WC columns each: the (re, im) of the outputs), and
// D = [D_0 .. D_7] holds the sums of equal weight in TMEM: A_i times the first 8 - i
// blocks adds into D_i .. D_7, so a K step of a tile takes eight MMAs of N = WC (8 - i).
// A thread reads its fibre's sums back, joins and rounds them: no shuffles, no fragments
// in registers; the outputs too small for the digits' bound it sums again in FP64.  Bound
// by the instructions that scale, cut and join (about 50 per complex number on either
// side) at the occupancy that registers and TMEM leave.  The products of the 8-SPF QVC
// model's EOM take 229 us (271 with mma.sync), of which 38 are for the scaling and the
// test of the outputs; with 12 SPFs 2,560 (3,230) and 350.
// ---------------------------------------------------------------------------
template <int NG>   // groups of four j
struct DigitTile {
  static constexpr int K = NG <= 2 ? 16 : 32;    // halfs per row
  static constexpr int WC = NG <= 2 ? 16 : 32;   // columns per weight
  static constexpr uint32_t SBO = K / 8 * 128, A = 128 * K * 2, B = 8 * WC * K * 2;
  static constexpr uint32_t COLS = 8 * WC;       // TMEM columns
  static constexpr uint32_t SMEM = 8 * A + B;
};
// The outputs of a fibre whose T = sum |x||m| does not show the digits to be accurate, from
// the leading ones in shared memory: a row of A_0, A_1 and the re columns of B_0, B_1.
template <int NG>
static __device__ __noinline__ unsigned digits_low(const unsigned char* a, const unsigned char* b, int nout) {
  using T = DigitTile<NG>;
  float x[4 * NG], any = 0.f;
#pragma unroll
  for (int k = 0; k < NG; ++k) {
    const uint4 u = *reinterpret_cast<const uint4*>(a + k * 128), v = *reinterpret_cast<const uint4*>(a + T::A + k * 128);
    x[4 * k] = fx_lead_sum(u.x, v.x);
    x[4 * k + 1] = fx_lead_sum(u.y, v.y);
    x[4 * k + 2] = fx_lead_sum(u.z, v.z);
    x[4 * k + 3] = fx_lead_sum(u.w, v.w);
    any += x[4 * k] + x[4 * k + 1] + x[4 * k + 2] + x[4 * k + 3];
  }
  if (any == 0.f) return 0u;   // a fibre of zeros
  unsigned low = 0u;
#pragma unroll 1
  for (int o = 0; o < nout; ++o) {
    const int n0 = 2 * o, n1 = T::WC + 2 * o;
    const unsigned char* b0 = b + (n0 >> 3) * T::SBO + (n0 & 7) * 16;
    const unsigned char* b1 = b + (n1 >> 3) * T::SBO + (n1 & 7) * 16;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < NG; ++k) {
      const uint4 u = *reinterpret_cast<const uint4*>(b0 + k * 128), v = *reinterpret_cast<const uint4*>(b1 + k * 128);
      t = fmaf(x[4 * k], fx_lead_sum(u.x, v.x), t);
      t = fmaf(x[4 * k + 1], fx_lead_sum(u.y, v.y), t);
      t = fmaf(x[4 * k + 2], fx_lead_sum(u.z, v.z), t);
      t = fmaf(x[4 * k + 3], fx_lead_sum(u.w, v.w), t);
    }
    if (t < FX_LOW) low |= 1u << o;
  }
  return low;
}

template <int NG>
__global__ void __launch_bounds__(128, NG <= 2 ? 4 : 2)
    prod_digits_kernel(const ProdDesc* __restrict__ descs, int ndesc, long long ntiles, int* status) {
  using T = DigitTile<NG>;
  extern __shared__ __align__(128) unsigned char tc_smem[];   // A_0 .. A_7, B
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t s_tmem;
  __shared__ unsigned rowexp[4 * NG], colmag[4 * NG];
  __shared__ __align__(16) unsigned scale[4 * NG];
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5;
  long long t0 = ntiles * blockIdx.x / gridDim.x;
  const long long tend = ntiles * (blockIdx.x + 1) / gridDim.x;
  if (tid == 0) tc_bar_init(&bar, 1);
  if (warp == 0) tc_alloc(&s_tmem, T::COLS);
  if (NG == 3)   // the last K group of A stays zero
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<uint4*>(tc_smem + i * T::A + (tid >> 3) * T::SBO + 3 * 128 + (tid & 7) * 16) = make_uint4(0, 0, 0, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem, base = tc_smem_addr(tc_smem);
  uint32_t parity = 0;
  bool ok = true;
  int di = t0 < tend ? warp_find_desc(descs, ndesc, t0) : 0;
  for (; ok && t0 < tend; ++di) {
    const ProdDesc& d = descs[di];
    const int nin = d.nin, nout = d.nout, sh = fx_headroom(nin);
    const float pw = fx_pow2(sh);
    const unsigned L = (unsigned)d.L, nfib = (unsigned)(d.L * d.R);
    const long long dend = min(tend, d.block_start + (long long)((nfib + 127) / 128));
    const long long Lx = d.L * (nin - 1), Ly = d.L * (nout - 1);
    unsigned p = (unsigned)(t0 - d.block_start) * 128 + tid, r = p / L;
    cplx x[4 * NG];
    auto fetch = [&]() {   // element j of fibre (l, r): l + L (j + nin r) = p + Lx r + L j
      const cplx* xp = d.X + ((long long)p + Lx * r);
      const bool act = p < nfib;
#pragma unroll
      for (int j = 0; j < 4 * NG; ++j) {
        x[j] = mkc(0.0, 0.0);
        if (act && j < nin) x[j] = *xp;
        xp += L;
      }
    };
    fetch();
    // the matrix and the sample of the scaling are on their way together; then a row's
    // exponent, its digits
    constexpr int PM = (T::WC / 2 * (T::K / 2) + 127) / 128;
    cplx mv[PM];
#pragma unroll
    for (int i = 0; i < PM; ++i) {
      const int e = tid + 128 * i, jo = e / (T::K / 2), ji = e % (T::K / 2);
      mv[i] = mkc(0.0, 0.0);
      if (jo < nout && ji < nin) mv[i] = d.conjT ? cconj(d.M[ji + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * ji];
    }
    __syncthreads();   // B of the descriptor before is read (its MMAs are complete)
    if (tid < 4 * NG) rowexp[tid] = 0u;
    if (tid == 0) s_bad = 0;
    fx_column_sizes(d, colmag);
    __syncthreads();
    bool scaled;
    {   // every warp for itself: the same values
      const unsigned b = fx_column_scale(colmag, nin);
      if ((tid & 31) < 4 * NG) scale[tid & 31] = b;
      scaled = __any_sync(0xffffffffu, b);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PM; ++i) {
      const int e = tid + 128 * i, jo = e / (T::K / 2), ji = e % (T::K / 2);
      if (jo < nout && ji < nin) atomicMax(&rowexp[jo], fx_scaled_down(fx_mag(mv[i]), scale[ji]));
    }
    __syncthreads();
    if (tid < nout && !fx_ok(rowexp[tid])) s_bad = 1;
#pragma unroll
    for (int q = 0; q < PM; ++q) {
      const int e = tid + 128 * q, jo = e / (T::K / 2), ji = e % (T::K / 2);
      if (e >= T::WC / 2 * (T::K / 2)) break;
      const cplx m = mv[q];
      const unsigned eb = (jo < nout ? fx_ebits(rowexp[jo]) : fx_ebits(0u)) + (ji < nin ? scale[ji] : 0u);
      unsigned s[8];
      fx_digits(m.x, m.y, eb, eb, s);
      unsigned char* b = tc_smem + 8 * T::A + (ji >> 2) * 128 + (ji & 3) * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {   // columns re: (Mr, -Mi), im: (Mi, Mr)
        const int n = i * T::WC + 2 * jo;
        *reinterpret_cast<unsigned*>(b + (n >> 3) * T::SBO + (n & 7) * 16) = s[i] ^ 0x80000000u;
        *reinterpret_cast<unsigned*>(b + (n >> 3) * T::SBO + ((n & 7) + 1) * 16) = __byte_perm(s[i], s[i], 0x1032);
      }
    }
    for (; t0 < dend; ++t0) {
      if (scaled) {
#pragma unroll
        for (int k = 0; k < NG; ++k) {
          const uint4 b = reinterpret_cast<const uint4*>(scale)[k];
          x[4 * k] = fx_scale_up(x[4 * k], b.x);
          x[4 * k + 1] = fx_scale_up(x[4 * k + 1], b.y);
          x[4 * k + 2] = fx_scale_up(x[4 * k + 2], b.z);
          x[4 * k + 3] = fx_scale_up(x[4 * k + 3], b.w);
        }
      }
      unsigned mag = 0u;
#pragma unroll
      for (int j = 0; j < 4 * NG; ++j) mag = max(mag, fx_mag(x[j]));
      const unsigned eb = fx_ebits(mag);
      const unsigned ef = fx_exp(eb, 0u, 44 + sh);
      bool bad = !fx_ok(mag);
#pragma unroll
      for (int k = 0; k < NG; ++k) {
        unsigned s[4][8];
#pragma unroll
        for (int j = 0; j < 4; ++j) fx_digits(x[4 * k + j].x, x[4 * k + j].y, eb, eb, s[j]);
        unsigned char* a = tc_smem + (tid >> 3) * T::SBO + k * 128 + (tid & 7) * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<uint4*>(a + i * T::A) = make_uint4(s[0][i], s[1][i], s[2][i], s[3][i]);
      }
      tc_fence_smem();
      tc_fence_before();
      __syncthreads();
      bad = bad || s_bad;
      if (tid == 0) {
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < T::K / 16; ++ks)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            tc_mma_f16(tmem + i * T::WC, tc_smem_desc(base + i * T::A + ks * 256, 128, T::SBO),
                       tc_smem_desc(base + 8 * T::A + ks * 256, 128, T::SBO), tc_idesc_f16(128, T::WC * (8 - i)),
                       ks || i);
        tc_commit(&bar);
      }
      const unsigned pc = p, rc = r;
      if (t0 + 1 < dend) {
        p += 128;
        r = p / L;
        fetch();
      }
      // every thread polls; the verdict is made uniform
      ok = __syncthreads_and(tc_wait(&bar, parity));
      if (!ok) break;
      parity ^= 1;
      tc_fence_after();
      const bool act = pc < nfib;
      unsigned least = 0xffffffffu;   // below 2 fx_small_limit: an output may be too small for its digits
      cplx* y = d.Y + ((long long)pc + Ly * rc);
#pragma unroll
      for (int h = 0; h < NG; ++h) {
        if (4 * h >= nout) break;
        float c[8][8];
        tc_ld8x8(tmem + ((uint32_t)(warp * 32) << 16) + 8 * h, T::WC, c);
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          if (4 * h + o < nout) {
            const unsigned es = fx_ebits(rowexp[4 * h + o]) + ef;
            const long long re = fx_join(c, 2 * o, pw), im = fx_join(c, 2 * o + 1, pw);
            least = min(least, fx_small_word(re, im, fx_small_limit(sh)));
            if (act && !bad) y[(long long)L * (4 * h + o)] = mkc(fx_double(re, es), fx_double(im, es));
          }
        }
      }
      if (act && bad) {
        prod_fibre_fp64(d, pc - L * rc, rc);
      } else if (act && least < 2 * fx_small_limit(sh)) {
        const unsigned low = digits_low<NG>(tc_smem + (tid >> 3) * T::SBO + (tid & 7) * 16, tc_smem + 8 * T::A, nout);
        if (low) prod_outputs_fp64(d, pc, low, 0, 1);
      }
    }
    t0 = dend;
  }
  if (!ok && tid == 0) tc_gave_up(&bar, parity, status);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tc_dealloc(tmem, T::COLS);
  }
}

template <int NG>
static void prod_digits_go(const ProdDesc* d, int nd, long long nblocks, int nsm, int* status, cudaStream_t st) {
  using T = DigitTile<NG>;
  const long long grid = std::min<long long>(nblocks, (NG <= 2 ? 4LL : 2LL) * nsm);
  prod_digits_kernel<NG><<<(unsigned)grid, 128, T::SMEM, st>>>(d, nd, nblocks, status);
}
void launch_prod_digits_tc(const ProdDesc* d, int nd, long long nblocks, int maxn, int* status, cudaStream_t st) {
  const int nsm = sm_count();
  if (maxn <= 8) prod_digits_go<2>(d, nd, nblocks, nsm, status, st);
  else if (maxn <= 12) prod_digits_go<3>(d, nd, nblocks, nsm, status, st);
  else prod_digits_go<4>(d, nd, nblocks, nsm, status, st);
}

// pipeline stages of the tensor-core mode product (MACAW_GB300_TC_STAGES=1 or 2)
static int g_tc_stages = 1;
// smallest largest-SPF-count of a batch that single contexts send to the tensor
// cores (MACAW_GB300_TC_MIN_N or mctdh_tensor_core_config).  Default 17, i.e.
// none: on the benchmark model the FP32 CUDA-core kernel is faster at 8 and at
// 12 SPFs and its round-to-nearest sums drift less over long propagations.
static int g_tc_min_n = 17;

// Once per process (context creation calls it): the settings from the environment.
void tc_prepare() {
  static std::once_flag once;
  std::call_once(once, [] {
    const char* e = getenv("MACAW_GB300_TC_STAGES");
    g_tc_stages = (e && e[0] == '2') ? 2 : 1;
    const char* m = getenv("MACAW_GB300_TC_MIN_N");
    if (m && atoi(m) > 0) g_tc_min_n = atoi(m);
  });
}
cudaError_t configure_tc() {
  cudaError_t e = allow_smem(prod_tc_kernel, 2 * TC_NPART * (TC_ROWS * 2 * TC_MAXN * 4 + 2 * TC_MAXN * 2 * TC_MAXN * 4));
  if (e == cudaSuccess) e = allow_smem(prod_digits_kernel<2>, DigitTile<2>::SMEM);
  if (e == cudaSuccess) e = allow_smem(prod_digits_kernel<3>, DigitTile<3>::SMEM);
  if (e == cudaSuccess) e = allow_smem(prod_digits_kernel<4>, DigitTile<4>::SMEM);
  return e;
}

// Tensor-core path for FP32 products of nin, nout <= 16, from the threshold on
// (force: any size up to 16); false: not taken
bool launch_prod_tc(const ProdDesc* d_descs, int ndesc, long long nblocks, int maxn, int* status, cudaStream_t st,
                    bool force) {
  if (maxn > TC_MAXN || (!force && maxn < g_tc_min_n) || ndesc <= 0 || nblocks <= 0) return false;
  const int K = ((2 * maxn + 7) / 8) * 8;
  const int N = 2 * maxn <= 16 ? 16 : 32;
  const size_t stage = (size_t)TC_NPART * ((size_t)TC_ROWS * K * 4 + (size_t)N * K * 4);
  const int nstage = g_tc_stages;
  const size_t smem = stage * nstage;
  const int per_sm = std::max(1, std::min(8, (int)((220 * 1024) / smem)));
  const long long grid = std::min<long long>(nblocks, (long long)sm_count() * per_sm);
  prod_tc_kernel<<<(unsigned)grid, TC_ROWS, smem, st>>>(d_descs, ndesc, nblocks, K, N, nstage, status);
  return true;
}

// the timeout flag (cleared when `clear`), or -1 when it could not be read
int tc_timeout_flag(bool clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_timeout, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v) {
    const int z = 0;
    if (cudaMemcpyToSymbol(g_tc_timeout, &z, sizeof(int)) != cudaSuccess) return -1;
  }
  return v;
}

extern "C" int64_t mctdh_tensor_core_status(int64_t* enabled, int64_t* timeouts) {
  if (enabled) *enabled = tc_enabled() ? 1 : 0;
  if (timeouts) {
    const int v = tc_timeout_flag(true);
    if (v < 0) return MCTDH_ECUDA;
    *timeouts = v;
  }
  return MCTDH_OK;
}

int tc_config() { return 4 * std::min(g_tc_min_n, TC_MAXN + 1) + g_tc_stages; }

extern "C" int64_t mctdh_tensor_core_config(int64_t min_n, int64_t stages) {
  if (min_n < 0 || stages < 0 || stages > 2) return MCTDH_EARG;
  if (min_n > 0) g_tc_min_n = (int)min_n;
  if (stages > 0) g_tc_stages = (int)stages;
  return MCTDH_OK;
}
