// FP64 kernels of the G-MCTDH equation-of-motion path for sm_103a.
//
// The FP32 forms of the mode products and single-hole contractions (precision 1) and
// what the FP64-accurate ones (fixed.cu, tc.cu) are launched by; one-mode operators, sums
// of terms, regularised inverses, integrator stages.  FP64 is the scarce unit of this
// chip, so these kernels spend it only on the algebra the EOM needs, each fibre of a
// tensor is read once, and reductions are two-stage with a fixed summation order, so
// that reruns are bitwise identical.
#include <algorithm>
#include <atomic>

#include "kernels.cuh"
#include "fixed.cuh"
#include <stdio.h>
#include <stdlib.h>

// ---------------------------------------------------------------------------
// descriptor lookup: descriptors are sorted by block_start
// ---------------------------------------------------------------------------
template <typename D>
__device__ __forceinline__ int find_desc_at(const D* descs, int ndesc, long long b) {
  int lo = 0, hi = ndesc - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (descs[mid].block_start <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}
template <typename D>
__device__ __forceinline__ int find_desc(const D* descs, int ndesc) {
  return find_desc_at(descs, ndesc, (long long)blockIdx.x);
}

// ---------------------------------------------------------------------------
// Batched mode product in FP32 (Mult_HeM_MatV / Mult_GM_MatV,
// gmctdh_objects.f90:1407-1468; FP64 accuracy in fixed.cu)
// One thread owns one fibre (l, :, r): it reads the nin inputs once into
// registers and writes the nout outputs.  Bound by latency: descriptor, matrix and fibre
// were three dependent trips to memory with two barriers before 256 multiply-adds a
// thread; the fibre is now fetched first (nine products of 32,768 fibres of 8: 14.2 ->
// 13.9 us).
// ---------------------------------------------------------------------------
// FP32 products: the FP32-rounded x and M are multiplied and accumulated in FP32
// (~1e-7 relative; the split's correction products would sit at the accumulation's
// own rounding level), outputs complex FP32 (TF_F32) or FP64.
// Block `bb` of the batch (blockIdx.x of the plain launch; persistent CTAs walk
// the blocks).
template <int MAXN>
__device__ __forceinline__ void prod_block(const ProdDesc* __restrict__ descs, int ndesc, long long bb) {
  __shared__ __align__(16) cplxf Mh[MAXN * MAXN];   // Mh[j + MAXN jo]: two j per load
  const ProdDesc& d = descs[warp_find_desc(descs, ndesc, bb)];
  const int nin = d.nin, nout = d.nout;
  const long long p = (bb - d.block_start) * blockDim.x + threadIdx.x;
  const long long L = d.L, nfib = L * d.R;
  const bool act = p < nfib;
  long long l = 0, r = 0;
  if (act) fibre_lr(p, L, nfib, l, r);
  const long long xi0 = l + L * (long long)nin * r;
  cplx* y0 = d.Y + l + L * (long long)nout * r;
  const cplx alpha = d.alpha;
  // the fibre is on its way while the matrix is staged
  cplxf xh[MAXN];
#pragma unroll
  for (int j = 0; j < MAXN; ++j) {
    const float4 w = (act && j < nin) ? load_split(d.X, xi0 + L * j, d.xfmt) : make_float4(0.f, 0.f, 0.f, 0.f);
    xh[j] = make_float2(w.x + w.z, w.y + w.w);   // rounded to nearest
  }
  for (int e = threadIdx.x; e < nin * nout; e += blockDim.x) {
    int jo = e % nout, ji = e / nout;
    cplx v = d.conjT ? cconj(d.M[ji + (long long)d.ldm * jo]) : d.M[jo + (long long)d.ldm * ji];
    float hx, lx, hy, ly;
    split_d2f(v.x, hx, lx);
    split_d2f(v.y, hy, ly);
    Mh[ji + MAXN * jo] = make_float2(hx + lx, hy + ly);   // rounded to nearest
  }
  __syncthreads();
  if (!act) return;
  const bool unit_alpha = (alpha.x == 1.0 && alpha.y == 0.0);
  for (int jo = 0; jo < nout; ++jo) {
    cplxf acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < MAXN; j += 2) {
      const float4 m = *reinterpret_cast<const float4*>(Mh + j + MAXN * jo);
      if (j < nin) acc = cfmaf_(acc, make_float2(m.x, m.y), xh[j]);
      if (j + 1 < nin) acc = cfmaf_(acc, make_float2(m.z, m.w), xh[j + 1]);
    }
    if (d.yfmt == TF_F32) {   // 8-byte elements: index from the tensor's base
      reinterpret_cast<float2*>(d.Y)[l + L * ((long long)nout * r + jo)] = acc;
      continue;
    }
    const cplx accd = mkc(f2d_exact(acc.x), f2d_exact(acc.y));
    cplx v = unit_alpha ? accd : cmul(alpha, accd);
    if (d.accumulate) v = cadd(v, y0[L * jo]);
    y0[L * jo] = v;
  }
}

template <int MAXN>
__global__ void __launch_bounds__(128) prod_kernel(const ProdDesc* __restrict__ descs, int ndesc) {
  prod_block<MAXN>(descs, ndesc, (long long)blockIdx.x);
}

// Persistent form: gridDim.x CTAs walk the batch's blocks in a fixed stride.
template <int MAXN>
__global__ void __launch_bounds__(128) prod_kernel_persistent(const ProdDesc* __restrict__ descs, int ndesc,
                                                              long long nblocks) {
  for (long long bb = blockIdx.x; bb < nblocks; bb += gridDim.x) {
    prod_block<MAXN>(descs, ndesc, bb);
    __syncthreads();   // the block's shared operands are rewritten by the next one
  }
}

// tcgen05 kernels (tc.cu) may serve the mode products unless MACAW_GB300_TC=0 keeps
// them out (read once per process).
bool tc_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("MACAW_GB300_TC");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on == 1;
}

int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    known[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// prec 0 and 2: FP64 accuracy (fixed.cu); prec 1: FP32 products.
// tc: 0 CUDA-core kernel, 1 tensor cores from the configured SPF count on,
// 2 tensor cores for every size they take (the ensemble autotuner's candidate).
// persist > 0: at most that many persistent CTAs walk the blocks.
void launch_prod(const ProdDesc* d_descs, int ndesc, long long nblocks, int maxn, bool plain, int* status, cudaStream_t st,
                 int prec, int tc, int persist) {
  if (ndesc <= 0 || nblocks <= 0) return;
  if (prec != 1) {
    launch_prod_fx(d_descs, ndesc, nblocks, maxn, plain, status, st, persist);
    return;
  }
  if (tc && tc_enabled() && launch_prod_tc(d_descs, ndesc, nblocks, maxn, status, st, tc == 2)) return;
  // register arrays sized for the batch's largest SPF count: no dead unrolled
  // iterations and fewer registers (more resident warps) at 8 SPFs and below
  if (persist > 0 && nblocks > persist) {
    const unsigned g = (unsigned)persist;
    if (maxn <= 8) prod_kernel_persistent<8><<<g, 128, 0, st>>>(d_descs, ndesc, nblocks);
    else if (maxn <= 12) prod_kernel_persistent<12><<<g, 128, 0, st>>>(d_descs, ndesc, nblocks);
    else prod_kernel_persistent<MAXN_SPF><<<g, 128, 0, st>>>(d_descs, ndesc, nblocks);
    return;
  }
  const unsigned nb = (unsigned)nblocks;
  if (maxn <= 8) prod_kernel<8><<<nb, 128, 0, st>>>(d_descs, ndesc);
  else if (maxn <= 12) prod_kernel<12><<<nb, 128, 0, st>>>(d_descs, ndesc);
  else prod_kernel<MAXN_SPF><<<nb, 128, 0, st>>>(d_descs, ndesc);
}

// ---------------------------------------------------------------------------
// Batched single-hole contraction with FP32 sums (precision modes 3 and 6; the
// others in fixed.cu), first stage (gmctdh_objects.f90:452-457, :595-600): FP32
// operands (rounded to nearest), FP32 products and sums (~1e-7 relative), the
// block partials widened to FP64 for the deterministic reduction.
// Block b of a descriptor handles fibre tiles b, b + nblk, ...; every thread owns
// one (j1, j2) pair and a fibre group; groups are summed in shared memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void hole_block(const HoleDesc* __restrict__ descs, int ndesc, long long bb) {
  __shared__ int s_di;
  __shared__ float2 X1[HOLE_TILE * MAXN_SPF];
  __shared__ float2 Y1[HOLE_TILE * MAXN_SPF];
  __shared__ cplx red[HOLE_THREADS];
  if (threadIdx.x == 0) s_di = find_desc_at(descs, ndesc, bb);
  __syncthreads();
  const HoleDesc& d = descs[s_di];
  const int b = (int)(bb - d.block_start);
  const int n1 = d.n1, n2 = d.n2, npairs = n1 * n2;
  const long long L = d.L, nfib = d.L * d.R;
  const long long ntiles = (nfib + HOLE_TILE - 1) / HOLE_TILE;
  const int tid = threadIdx.x;
  const bool small = npairs <= HOLE_THREADS;
  const int G = small ? HOLE_THREADS / npairs : 1;
  const int pair0 = small ? tid % npairs : tid;
  const int g = small ? tid / npairs : 0;
  float ah[4][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  // Staging: thread tid always loads fibre q = tid % HOLE_TILE of a tile and the
  // columns j = tid / HOLE_TILE, + HOLE_THREADS / HOLE_TILE, ...; its fibre's
  // (l, r) is carried from tile to tile instead of divided out per element.
  static_assert(HOLE_THREADS % HOLE_TILE == 0, "staging assumes whole tiles per thread row");
  const int qt = tid % HOLE_TILE, jt = tid / HOLE_TILE, jstep = HOLE_THREADS / HOLE_TILE;
  long long pcur = (long long)b * HOLE_TILE + qt;
  long long lcur = pcur % L, rcur = pcur / L;
  const long long pstep = (long long)d.nblk * HOLE_TILE;
  const long long dl = pstep % L, dr = pstep / L;
  for (long long tile = b; tile < ntiles; tile += d.nblk) {
    const bool in_range = pcur < nfib;
    const long long xb = lcur + L * (long long)n1 * rcur, yb = lcur + L * (long long)n2 * rcur;
    pcur += pstep;
    lcur += dl;
    rcur += dr;
    if (lcur >= L) { lcur -= L; rcur += 1; }
    for (int j = jt; j < n1; j += jstep) {
      const float4 w = in_range ? load_split(d.X, xb + L * j, d.xfmt) : make_float4(0.f, 0.f, 0.f, 0.f);
      X1[qt * MAXN_SPF + j] = make_float2(w.x + w.z, w.y + w.w);
    }
    for (int j = jt; j < n2; j += jstep) {
      const float4 w = in_range ? load_split(d.Y, yb + L * j, d.yfmt) : make_float4(0.f, 0.f, 0.f, 0.f);
      Y1[qt * MAXN_SPF + j] = make_float2(w.x + w.z, w.y + w.w);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int pr, q0, qs;
      if (small) {
        if (k > 0 || g >= G) break;
        pr = pair0; q0 = g; qs = G;
      } else {
        pr = pair0 + HOLE_THREADS * k;
        if (pr >= npairs) break;
        q0 = 0; qs = 1;
      }
      const int j1 = pr % n1, j2 = pr / n1;
      for (int q = q0; q < HOLE_TILE; q += qs) {
        const float2 x = X1[q * MAXN_SPF + j1], y = Y1[q * MAXN_SPF + j2];
        ah[k][0] = fmaf(x.x, y.x, ah[k][0]);
        ah[k][0] = fmaf(x.y, y.y, ah[k][0]);
        ah[k][1] = fmaf(x.x, y.y, ah[k][1]);
        ah[k][1] = fmaf(-x.y, y.x, ah[k][1]);
      }
    }
    __syncthreads();
  }
  cplx acc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) acc[k] = mkc(f2d_exact(ah[k][0]), f2d_exact(ah[k][1]));
  cplx* out = d.partial + (long long)b * npairs;
  if (small) {
    red[tid] = acc[0];
    __syncthreads();
    if (tid < npairs) {
      cplx s = mkc(0, 0);
      for (int gg = 0; gg < G; ++gg) s = cadd(s, red[gg * npairs + tid]);
      out[tid] = s;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int pr = pair0 + HOLE_THREADS * k;
      if (pr < npairs) out[pr] = acc[k];
    }
  }
}

__global__ void __launch_bounds__(HOLE_THREADS, 4) hole_kernel(const HoleDesc* __restrict__ descs, int ndesc) {
  hole_block(descs, ndesc, (long long)blockIdx.x);
}

// Persistent form: gridDim.x CTAs walk the batch's blocks in a fixed stride (each
// block still writes its own partial, so the sums do not depend on the grid).
__global__ void __launch_bounds__(HOLE_THREADS, 4) hole_kernel_persistent(const HoleDesc* __restrict__ descs,
                                                                       int ndesc, long long nblocks) {
  for (long long bb = blockIdx.x; bb < nblocks; bb += gridDim.x) {
    hole_block(descs, ndesc, bb);
    __syncthreads();   // the staging tiles are rewritten by the next block
  }
}

// prec 1: FP32 sums, else FP64 accuracy (fixed.cu)
void launch_hole(const HoleLaunch& b, cudaStream_t st, int prec, int persist) {
  if (b.ndesc <= 0 || b.nblocks <= 0) return;
  if (prec != 1) {
    launch_hole_fx(b, st, persist);
    return;
  }
  if (persist > 0 && b.nblocks > persist)
    hole_kernel_persistent<<<(unsigned)persist, HOLE_THREADS, 0, st>>>(b.d, b.ndesc, b.nblocks);
  else
    hole_kernel<<<(unsigned)b.nblocks, HOLE_THREADS, 0, st>>>(b.d, b.ndesc);
}

// ---------------------------------------------------------------------------
// Second stage: deterministic sum of partials into the target matrices.
// ---------------------------------------------------------------------------
// One block per target; the partial blocks of every term are spread over G thread
// groups (G = blockDim / (n1 n2) when that is > 1), each group sums its share in a
// fixed order, then the groups are added in group order (deterministic).
__global__ void __launch_bounds__(256) reduce_kernel(const RedTarget* __restrict__ tg,
                                                     const RedTerm* __restrict__ terms) {
  __shared__ cplx red[256], redT[256];
  const RedTarget& t = tg[blockIdx.x];
  const int npairs = t.n1 * t.n2;
  const int G = (npairs <= (int)blockDim.x / 2) ? (int)blockDim.x / npairs : 1;
  const int g = (G > 1) ? (int)threadIdx.x / npairs : 0;
  const int p0 = (G > 1) ? (int)threadIdx.x % npairs : (int)threadIdx.x;
  for (int base = 0; base < npairs; base += (G > 1 ? npairs : (int)blockDim.x)) {
    const int pr = base + p0;
    const bool act = (G > 1) ? (g < G) : (pr < npairs);
    cplx s = mkc(0, 0), sT = mkc(0, 0);
    if (act) {
      const int j1 = pr % t.n1, j2 = pr / t.n1;
      const int prT = j2 + t.n1 * j1;
      const int prC = j2 + t.n2 * j1;   // element (j2, j1) of an n2 x n1 source (conjT terms)
      for (int k = 0; k < t.count; ++k) {
        const RedTerm& rt = terms[t.first + k];
        cplx a = mkc(0, 0), aT = mkc(0, 0);
        for (int bb = g; bb < rt.nblk; bb += G) {
          if (rt.conjT) {
            a = cadd(a, cconj(rt.partial[(long long)bb * npairs + prC]));
            if (t.hermitize) aT = cadd(aT, cconj(rt.partial[(long long)bb * npairs + pr]));
          } else {
            a = cadd(a, rt.partial[(long long)bb * npairs + pr]);
            if (t.hermitize) aT = cadd(aT, rt.partial[(long long)bb * npairs + prT]);
          }
        }
        s = cadd(s, cmul(rt.alpha, a));
        if (t.hermitize) sT = cadd(sT, cmul(rt.alpha, aT));
      }
    }
    if (G > 1) {
      red[threadIdx.x] = s;
      redT[threadIdx.x] = sT;
      __syncthreads();
      if (g == 0) {
        for (int q = 1; q < G; ++q) {
          s = cadd(s, red[q * npairs + p0]);
          sT = cadd(sT, redT[q * npairs + p0]);
        }
      }
      __syncthreads();
    }
    if (act && g == 0) {
      const int j1 = pr % t.n1, j2 = pr / t.n1;
      if (t.hermitize) s = cscale(cadd(s, cconj(sT)), 0.5);
      cplx* o = t.out + j1 + (long long)t.ld * j2;
      *o = t.accumulate ? cadd(*o, s) : s;
    }
  }
}

void launch_reduce(const RedTarget* d_tg, int ntg, const RedTerm* d_terms, cudaStream_t st) {
  if (ntg <= 0) return;
  reduce_kernel<<<ntg, 256, 0, st>>>(d_tg, d_terms);
}

// ---------------------------------------------------------------------------
// h1mode and operator-applied SPFs for DVR modes (Calc_h1mode, hamilton.f90:416-482;
// MultTens / MultTensDiag, :577-629).  One block per (mode, operator).
// ---------------------------------------------------------------------------
// One block per (operator, SPF column j2): the primitive DOF operators act
// within each SPF, so a column is transformed in shared memory on its own
// (MultTens / MultTensDiag, hamilton.f90:577-629).  The DVR matrices of p, qp
// (i x real) and d^2/dq^2 (real) are applied with real arithmetic.  The operators with
// such matrices cost 2 ng FP64 instructions per element and come first in the list, the
// columns of an operator as neighbouring blocks, so that the SMs share them evenly.
// project: also the column j2 of phi_l^H (O phi_r), one warp per row j1 (small models;
// H1_PROJECT_MIN).
__global__ void __launch_bounds__(256) h1_kernel(const H1Desc* __restrict__ descs, int maxn2, bool project) {
  extern __shared__ cplx sm[];
  const H1Desc& d = descs[blockIdx.x / maxn2];
  const int j2 = blockIdx.x % maxn2;
  if (j2 >= d.n2) return;
  const int G = d.G, n1 = d.n1;
  cplx* bufA = sm;
  cplx* bufB = sm + G;
  const cplx* src = d.phi_r + (long long)G * j2;
  for (int e = threadIdx.x; e < G; e += blockDim.x) bufA[e] = src[e];
  __syncthreads();
  int ll = 1;
  for (int k = 0; k < d.ndof; ++k) {
    const int ng = d.ng[k];
    const int ot = d.optype[k];
    if (ot != 0) {
      const cplx* M = d.mat[k];
      for (int e = threadIdx.x; e < G; e += blockDim.x) {
        const int a = e % ll;
        const int gg = (e / ll) % ng;
        const int bidx = e / (ll * ng);
        cplx v;
        if (ot == 2) {
          v = cscale(bufA[e], M[gg].x);
        } else {
          // psi(.., g, ..) <- sum_g' psi(.., g', ..) M(g', g)   (zlacrm from the right)
          const cplx* in = bufA + a + (long long)ll * ng * bidx;
          const cplx* mc = M + (long long)ng * gg;
          double sx = 0.0, sy = 0.0;
          if (ot == 1) {
            for (int gp = 0; gp < ng; ++gp) {
              const cplx x = in[(long long)ll * gp];
              sx = fma(mc[gp].x, x.x, sx);
              sy = fma(mc[gp].x, x.y, sy);
            }
            v = mkc(sx, sy);
          } else {
            for (int gp = 0; gp < ng; ++gp) {
              const cplx x = in[(long long)ll * gp];
              sx = fma(mc[gp].y, x.x, sx);
              sy = fma(mc[gp].y, x.y, sy);
            }
            v = mkc(-sy, sx);   // i * (real matrix x column)
          }
        }
        bufB[e] = v;
      }
      __syncthreads();
      cplx* t = bufA; bufA = bufB; bufB = t;
    }
    ll *= ng;
  }
  cplx* dst = d.ophi + (long long)G * j2;
  for (int e = threadIdx.x; e < G; e += blockDim.x) dst[e] = bufA[e];
  if (!project) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j1 = warp; j1 < n1; j1 += (int)(blockDim.x >> 5)) {
    const cplx* pl = d.phi_l + (long long)G * j1;
    cplx s = mkc(0, 0);
    for (int gg = lane; gg < G; gg += 32) cfma_conj(s, pl[gg], bufA[gg]);
    for (int o = 16; o > 0; o >>= 1) {
      s.x += __shfl_down_sync(0xffffffffu, s.x, o);
      s.y += __shfl_down_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) {
      if (d.same_state) d.X[j1 + n1 * j2] = s;
      else d.h[j1 + n1 * j2] = s;
    }
  }
}

// acc (hi, lo) += a * b for FP32 pairs a = ah + al, b = bh + bl: the leading
// product is split exactly with an FMA, the sum keeps its rounding error in lo.
__device__ __forceinline__ void df_fma(float& sh, float& sl, float ah, float al, float bh, float bl) {
  const float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, e);
  e = fmaf(al, bh, e);
  const float s = sh + p;
  const float bp = s - sh;
  const float t = (sh - (s - bp)) + (p - bp);
  sh = s;
  sl += t + e;
}

// Split-FP32 variant of h1_kernel, for contexts with FP32 mode products: the column is held
// as FP32 (hi, lo) pairs, the DOF matrices come pre-split, every product is
// accumulated as a compensated FP32 pair (df_fma, ~1e-13 relative).  FP32 products round
// the operators' matrices to FP32: another 1e-13 in them now and then rounds an element the
// other way, 6e-8 of it, so these contexts keep one arithmetic for them (the FP64 forms
// are as fast: 62 us for 12 SPFs against 26 and 33).
__global__ void __launch_bounds__(256) h1_split_kernel(const H1Desc* __restrict__ descs, int maxn2, bool project) {
  extern __shared__ float4 smf[];
  const H1Desc& d = descs[blockIdx.x / maxn2];
  const int j2 = blockIdx.x % maxn2;
  if (j2 >= d.n2) return;
  const int G = d.G, n1 = d.n1;
  float4* bufA = smf;
  float4* bufB = smf + G;
  const cplx* src = d.phi_r + (long long)G * j2;
  for (int e = threadIdx.x; e < G; e += blockDim.x) {
    const cplx v = src[e];
    float hx, lx, hy, ly;
    split_d2f(v.x, hx, lx);
    split_d2f(v.y, hy, ly);
    bufA[e] = make_float4(hx, hy, lx, ly);
  }
  __syncthreads();
  int ll = 1;
  for (int k = 0; k < d.ndof; ++k) {
    const int ng = d.ng[k];
    const int ot = d.optype[k];
    if (ot != 0) {
      const float2* Mf = d.matf[k];
      for (int e = threadIdx.x; e < G; e += blockDim.x) {
        const int a = e % ll;
        const int gg = (e / ll) % ng;
        const int bidx = e / (ll * ng);
        float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
        if (ot == 2) {
          const float4 x = bufA[e];
          const float2 m = Mf[gg];
          df_fma(rh, rl, m.x, m.y, x.x, x.z);
          df_fma(ih, il, m.x, m.y, x.y, x.w);
        } else {
          const float4* in = bufA + a + (long long)ll * ng * bidx;
          const float2* mc = Mf + (long long)ng * gg;
          for (int gp = 0; gp < ng; ++gp) {
            const float4 x = in[(long long)ll * gp];
            const float2 m = mc[gp];
            df_fma(rh, rl, m.x, m.y, x.x, x.z);
            df_fma(ih, il, m.x, m.y, x.y, x.w);
          }
        }
        bufB[e] = (ot == 3) ? make_float4(-ih, rh, -il, rl) : make_float4(rh, ih, rl, il);
      }
      __syncthreads();
      float4* t = bufA; bufA = bufB; bufB = t;
    }
    ll *= ng;
  }
  cplx* dst = d.ophi + (long long)G * j2;
  for (int e = threadIdx.x; e < G; e += blockDim.x) {
    const float4 x = bufA[e];
    dst[e] = mkc(f2d_exact(x.x) + f2d_exact(x.z), f2d_exact(x.y) + f2d_exact(x.w));
  }
  if (!project) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j1 = warp; j1 < n1; j1 += (int)(blockDim.x >> 5)) {
    const cplx* pl = d.phi_l + (long long)G * j1;
    float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
    for (int gg = lane; gg < G; gg += 32) {
      const cplx p = pl[gg];
      float phx, plx, phy, ply;
      split_d2f(p.x, phx, plx);
      split_d2f(p.y, phy, ply);
      const float4 x = bufA[gg];
      // conj(p) * x
      df_fma(rh, rl, phx, plx, x.x, x.z);
      df_fma(rh, rl, phy, ply, x.y, x.w);
      df_fma(ih, il, phx, plx, x.y, x.w);
      df_fma(ih, il, -phy, -ply, x.x, x.z);
    }
    cplx s = mkc(f2d_exact(rh) + f2d_exact(rl), f2d_exact(ih) + f2d_exact(il));
    for (int o = 16; o > 0; o >>= 1) {
      s.x += __shfl_down_sync(0xffffffffu, s.x, o);
      s.y += __shfl_down_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) {
      if (d.same_state) d.X[j1 + n1 * j2] = s;
      else d.h[j1 + n1 * j2] = s;
    }
  }
}

// Blocks 0 .. nh - 1: same-state h1mode = (X + X^H) / 2 (the zher2k form,
// hamilton.f90:500-506).  The others: operators pre-summed per state and mode,
// out = sum_k coeff_k src_k, from the same X.
__global__ void h1_finish_kernel(const H1Desc* __restrict__ descs, int nh, const MatSumDesc* __restrict__ sums,
                                 const MatSumSrc* __restrict__ srcs) {
  if ((int)blockIdx.x >= nh) {
    const MatSumDesc& m = sums[blockIdx.x - nh];
    for (int e = threadIdx.x; e < m.n1 * m.n2; e += blockDim.x) {
      const int j1 = e % m.n1, j2 = e / m.n1, eT = j2 + m.n1 * j1;
      cplx acc = mkc(0, 0);
      for (int k = 0; k < m.count; ++k) {
        const MatSumSrc& x = srcs[m.first + k];
        cplx v = x.src[e];
        if (x.herm) v = cscale(cadd(v, cconj(x.src[eT])), 0.5);
        cfma(acc, x.coeff, v);
      }
      m.out[e] = acc;
    }
    return;
  }
  const H1Desc& d = descs[blockIdx.x];
  if (!d.same_state) return;
  const int n1 = d.n1;
  for (int pr = threadIdx.x; pr < n1 * d.n2; pr += blockDim.x) {
    const int j1 = pr % n1, j2 = pr / n1;
    d.h[pr] = cscale(cadd(d.X[pr], cconj(d.X[j2 + n1 * j1])), 0.5);
  }
}

cudaError_t prepare_device() {
  cudaError_t e = allow_smem(h1_kernel, 227 * 1024);
  if (e == cudaSuccess) e = allow_smem(h1_split_kernel, 227 * 1024);
  if (e == cudaSuccess) e = configure_fx();
  if (e == cudaSuccess) e = configure_spf();
  if (e == cudaSuccess) e = configure_tc();
  return e;
}

int launch_h1(const H1Launch& b, bool with_h, cudaStream_t st, const MatSumDesc* sums, int nsums,
              const MatSumSrc* srcs) {
  int launches = 0;
  const bool proj = with_h && b.proj.ndesc > 0;
  if (b.n > 0) {
    if (b.split) h1_split_kernel<<<(unsigned)(b.n * b.maxn2), 256, b.smem, st>>>(b.d, b.maxn2, with_h);
    else h1_kernel<<<(unsigned)(b.n * b.maxn2), 256, b.smem, st>>>(b.d, b.maxn2, with_h && !proj);
    ++launches;
  }
  if (proj) {
    launch_hole(b.proj, st);
    ++launches;
  }
  const int nh = with_h ? b.n : 0;
  if (nh + nsums > 0) {
    h1_finish_kernel<<<nh + nsums, 128, 0, st>>>(b.d, nh, sums, srcs);
    ++launches;
  }
  return launches;
}

// ---------------------------------------------------------------------------
// Parallel complex Jacobi eigen-decomposition of a Hermitian matrix (n <= 32)
// held in shared memory, run by one warp: the work zheev does inside StdRegInv
// (maths.f90:36).  Each round rotates the n/2 disjoint index pairs of a
// round-robin schedule at once (column rotations A J, then row rotations J^H (A J);
// rotations of disjoint pairs commute), so a sweep is n-1 rounds.  A pair is
// rotated when |a_pq|^2 > 1e-38 ||A||_F^2 and |a_pq|^2 > 1e-32 |a_pp a_qq|; the
// sweep count is capped.  A[i + ld*j], V likewise.  *ok: the sweeps converged.
// ---------------------------------------------------------------------------
#define JAC_MAX_SWEEPS 40
struct JacRot {
  double c, s, tm, app, aqq;
  cplx u;
  int p, q, rot;
};

__device__ void jacobi_herm(cplx* A, cplx* V, int n, int ld, JacRot* R, bool* ok) {
  const int lane = threadIdx.x;   // blockDim.x == 32
  for (int e = lane; e < n * n; e += 32) {
    int i = e % n, j = e / n;
    V[i + ld * j] = mkc(i == j ? 1.0 : 0.0, 0.0);
  }
  __syncwarp();
  double fro2 = 0.0;
  for (int e = 0; e < n * n; ++e) { int i = e % n, j = e / n; fro2 += cabs2(A[i + ld * j]); }
  const int m = n + (n & 1);      // even count; index n is a dummy for odd n
  const int npair = m / 2;
  bool converged = (n <= 1);
  for (int sweep = 0; sweep < JAC_MAX_SWEEPS && !converged; ++sweep) {
    bool any = false;
    for (int r = 0; r < m - 1; ++r) {
      int rot = 0;
      if (lane < npair) {
        // circle schedule: (r, m-1) and ((r+j) mod (m-1), (r-j) mod (m-1))
        int a = (lane == 0) ? r : (r + lane) % (m - 1);
        int b = (lane == 0) ? m - 1 : (r - lane + (m - 1)) % (m - 1);
        const int p = min(a, b), q = max(a, b);
        JacRot& J = R[lane];
        J.p = p;
        J.q = q;
        if (q < n) {
          const cplx apq = A[p + ld * q];
          const double m2 = cabs2(apq);
          const double app = A[p + ld * p].x, aqq = A[q + ld * q].x;
          rot = (m2 > 1e-38 * fro2) && (m2 > 1e-32 * fabs(app * aqq));
          if (rot) {
            // one reciprocal square root for |a_pq| (the FP64 pipe is the bottleneck here)
            const double rm = rsqrt(m2);
            const double mag = m2 * rm;
            const double tau = (aqq - app) * 0.5 * rm;
            const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            J.c = rsqrt(1.0 + t * t);
            J.s = t * J.c;
            J.u = mkc(apq.x * rm, apq.y * rm);
            J.tm = t * mag;
            J.app = app;
            J.aqq = aqq;
          }
        }
        J.rot = rot;
      }
      const unsigned ballot = __ballot_sync(0xffffffffu, rot);
      __syncwarp();
      if (ballot == 0) continue;
      any = true;
      // column rotations: work items (row, pair) spread over the lanes (one item per
      // lane for n <= 8); pairs are disjoint, so items never share an element
      for (int it = lane; it < n * npair; it += 32) {
        const int row = it % n;
        const JacRot& J = R[it / n];
        if (!J.rot) continue;
        const cplx uc = cconj(J.u);
        cplx ap = A[row + ld * J.p], aq = A[row + ld * J.q];
        A[row + ld * J.p] = csub(cscale(ap, J.c), cscale(cmul(uc, aq), J.s));
        A[row + ld * J.q] = cadd(cscale(cmul(J.u, ap), J.s), cscale(aq, J.c));
        cplx vp = V[row + ld * J.p], vq = V[row + ld * J.q];
        V[row + ld * J.p] = csub(cscale(vp, J.c), cscale(cmul(uc, vq), J.s));
        V[row + ld * J.q] = cadd(cscale(cmul(J.u, vp), J.s), cscale(vq, J.c));
      }
      __syncwarp();
      // row rotations: items (column, pair)
      for (int it = lane; it < n * npair; it += 32) {
        const int col = it % n;
        const JacRot& J = R[it / n];
        if (!J.rot) continue;
        cplx ap = A[J.p + ld * col], aq = A[J.q + ld * col];
        A[J.p + ld * col] = csub(cscale(ap, J.c), cscale(cmul(J.u, aq), J.s));
        A[J.q + ld * col] = cadd(cscale(cmul(cconj(J.u), ap), J.s), cscale(aq, J.c));
      }
      __syncwarp();
      // the rotated 2x2 blocks in closed form (other pairs never touch them)
      if (lane < npair && rot) {
        const JacRot& J = R[lane];
        A[J.p + ld * J.p] = mkc(J.app - J.tm, 0.0);
        A[J.q + ld * J.q] = mkc(J.aqq + J.tm, 0.0);
        A[J.p + ld * J.q] = mkc(0, 0);
        A[J.q + ld * J.p] = mkc(0, 0);
      }
      __syncwarp();
    }
    converged = !any;
  }
  *ok = converged;
}

// Inverse of a Hermitian positive definite n x n matrix (n <= 32) by n symmetric sweeps
// (Gauss-Jordan elimination of the upper triangle, whose every intermediate is
// Hermitian): A -> A^-1 in place, A[i + ld j], both triangles filled.  A thread holds EPT
// elements of the triangle; per sweep one column passes through shared memory
// (v, two buffers of 32).  One sweep costs a reciprocal and six dependent FP64
// instructions, against the rotations of six to ten Jacobi sweeps of n - 1 rounds.
// Returns false (on every thread) at a pivot that is not positive; all threads call it.
template <int EPT>
__device__ __forceinline__ bool sweep_inverse(cplx* A, int n, int ld, cplx (*v)[MAXN_SPF]) {
  cplx a[EPT];
  int ei[EPT], ej[EPT];
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    int e = threadIdx.x + q * blockDim.x, j = 0;
    if (e >= n * (n + 1) / 2) {
      ei[q] = ej[q] = -1;
      a[q] = mkc(0, 0);
      continue;
    }
    while (e > j) e -= ++j;   // e -> (i <= j), j-major
    ei[q] = e;
    ej[q] = j;
    a[q] = A[e + ld * j];
    if (e == 0) v[0][j] = cconj(a[q]);
  }
  bool ok = true;
  for (int k = 0; k < n; ++k) {
    __syncthreads();
    const cplx* vk = v[k & 1];
    const double d = vk[k].x;
    ok = ok && d > 0.0;
    const double p = newton_rcp(d);
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
      const int i = ei[q], j = ej[q];
      if (i < 0) continue;
      const bool row = i == k, col = j == k;
      const cplx vj = vk[j];
      const cplx w = cscale(row ? cconj(vj) : vk[i], p);
      if (row || col) {
        a[q] = (row && col) ? mkc(-p, 0.0) : w;
      } else {
        a[q].x = fma(-w.x, vj.x, fma(-w.y, vj.y, a[q].x));
        a[q].y = fma(-w.y, vj.x, fma(w.x, vj.y, a[q].y));
        if (i == j) a[q].y = 0.0;
      }
      if (i == k + 1) v[(k + 1) & 1][j] = cconj(a[q]);
      else if (j == k + 1) v[(k + 1) & 1][i] = a[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    if (ei[q] < 0) continue;
    A[ei[q] + ld * ej[q]] = mkc(-a[q].x, -a[q].y);
    A[ej[q] + ld * ei[q]] = mkc(-a[q].x, a[q].y);
  }
  __syncthreads();
  return ok;
}

// Where every eigenvalue of rho is at least eps the 'poly' regularisation is the plain
// inverse, 1 / w; the inverse itself shows it: positive pivots, and eps |rho^-1|_F <= 1
// bounds its largest eigenvalue.  Then no eigen-decomposition is needed (8 x 8: 63 -> 9 us
// a launch of 18 matrices); otherwise the Jacobi path below.  blockIdx.y: the blocks
// of a matrix share its rho^-1 MF products, one warp per operator at a time, each
// inverting for itself.
//
// Jacobi path: four warps per (mode, state), the sweeps on the first (its
// rotations are one round per warp-wide step), the warm-start products, the
// regularised inverse and the rho^-1 MF products on all four (independent
// FP64 dot products, so more of them in flight against the FP64 latency).
__global__ void __launch_bounds__(128) reginv_kernel(const RegInvDesc* __restrict__ descs, const MFOp* __restrict__ ops,
                                                     int* status) {
  __shared__ cplx A[MAXN_SPF * MAXN_SPF];
  __shared__ cplx V[MAXN_SPF * MAXN_SPF];
  __shared__ cplx Inv[MAXN_SPF * MAXN_SPF];
  __shared__ double w[MAXN_SPF];
  __shared__ JacRot R[MAXN_SPF / 2];
  __shared__ cplx vcol[2][MAXN_SPF];
  __shared__ float fro[4];
  const RegInvDesc& d = descs[blockIdx.x];
  const int n = d.n, ld = MAXN_SPF;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    // upper triangle is authoritative (zheev 'U'): mirror it
    cplx v = (i <= j) ? d.A[i + n * j] : cconj(d.A[j + n * i]);
    if (i == j) v.y = 0.0;
    A[i + ld * j] = v;
    Inv[i + ld * j] = v;
  }
  __syncthreads();
  if (d.regtype == 0) {
    const bool pos = n <= 15 ? sweep_inverse<1>(Inv, n, ld, vcol) : sweep_inverse<5>(Inv, n, ld, vcol);
    float f2 = 0.f;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const cplx v = Inv[e % n + ld * (e / n)];
      const float x = (float)(v.x * d.eps), y = (float)(v.y * d.eps);   // about one at most, whatever eps
      f2 = fmaf(x, x, fmaf(y, y, f2));
    }
    for (int o = 16; o > 0; o >>= 1) f2 += __shfl_down_sync(0xffffffffu, f2, o);
    if ((threadIdx.x & 31) == 0) fro[threadIdx.x >> 5] = f2;
    __syncthreads();
    if (pos && fro[0] + fro[1] + fro[2] + fro[3] <= 0.998f) {
      if (d.inv_out && blockIdx.y == 0)
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) d.inv_out[e] = Inv[e % n + ld * (e / n)];
      const int lane = threadIdx.x & 31;
      for (int o = blockIdx.y * 4 + (threadIdx.x >> 5); o < d.op_count; o += 4 * gridDim.y) {
        const MFOp& op = ops[d.op_first + o];
        for (int e = lane; e < n * op.n2; e += 32) {
          const int i = e % n, j = e / n;
          cplx s = mkc(0, 0);
          for (int k = 0; k < n; ++k) cfma(s, Inv[i + ld * k], op.mf[k + n * j]);
          op.out[e] = s;
        }
      }
      return;
    }
  }
  if (blockIdx.y > 0) return;   // the first block's alone (it keeps the warm-start vectors)
  // Warm start: rho changes little between consecutive calls (the mean-field
  // evaluations of one propagation), so the previous eigenvectors Vp nearly
  // diagonalise it; Jacobi then runs on Vp^H A Vp and the eigenvectors are Vp V.
  // The same eigen-decomposition up to rounding, in one or two sweeps instead of
  // a cold start's six to ten.  Every 64th call starts cold, which bounds the
  // drift of the accumulated product from unitarity.
  const int wcount = d.vprev ? *d.vcount : 0;
  const bool warm = wcount > 0 && wcount < 64;
  if (warm) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {   // Inv <- A Vp
      const int i = e % n, j = e / n;
      cplx s = mkc(0, 0);
      for (int k = 0; k < n; ++k) cfma(s, A[i + ld * k], d.vprev[k + n * j]);
      Inv[i + ld * j] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {   // V <- Vp^H Inv
      const int i = e % n, j = e / n;
      cplx s = mkc(0, 0);
      for (int k = 0; k < n; ++k) cfma_conj(s, d.vprev[k + n * i], Inv[k + ld * j]);
      V[i + ld * j] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {   // Hermitian from the upper triangle
      const int i = e % n, j = e / n;
      cplx v = (i <= j) ? V[i + ld * j] : cconj(V[j + ld * i]);
      if (i == j) v.y = 0.0;
      A[i + ld * j] = v;
    }
    __syncthreads();
  }
  bool ok = true;
  if (threadIdx.x < 32) jacobi_herm(A, V, n, ld, R, &ok);
  __syncthreads();
  if (!ok && threadIdx.x == 0) atomicOr(status, DEVST_EIG_NOCONV);
  if (warm) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {   // Inv <- Vp V
      const int i = e % n, j = e / n;
      cplx s = mkc(0, 0);
      for (int k = 0; k < n; ++k) cfma(s, d.vprev[i + n * k], V[k + ld * j]);
      Inv[i + ld * j] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) V[e % n + ld * (e / n)] = Inv[e % n + ld * (e / n)];
    __syncthreads();
  }
  if (d.vprev) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) d.vprev[e] = V[e % n + ld * (e / n)];
    if (threadIdx.x == 0) *d.vcount = (warm && ok) ? wcount + 1 : (ok ? 1 : 0);
  }
  if (threadIdx.x < n) {
    double wv = A[threadIdx.x + ld * threadIdx.x].x;
    double f;
    if (d.regtype == 0) {   // 'poly'
      double eps = d.eps;
      double wr = (wv < eps) ? 0.5 * (eps + wv * wv / eps) : wv;
      f = 1.0 / wr;
    } else {                // 'tikh'
      f = wv / (wv * wv + d.eps * d.eps);
    }
    w[threadIdx.x] = f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    cplx s = mkc(0, 0);
    for (int k = 0; k < n; ++k) {
      cplx vik = V[i + ld * k], vjk = V[j + ld * k];
      s = cadd(s, cscale(cmul(vik, cconj(vjk)), w[k]));
    }
    Inv[i + ld * j] = s;
    if (d.inv_out) d.inv_out[i + n * j] = s;
  }
  __syncthreads();
  for (int o = 0; o < d.op_count; ++o) {
    const MFOp& op = ops[d.op_first + o];
    for (int e = threadIdx.x; e < n * op.n2; e += blockDim.x) {
      int i = e % n, j = e / n;
      cplx s = mkc(0, 0);
      for (int k = 0; k < n; ++k) cfma(s, Inv[i + ld * k], op.mf[k + n * j]);
      op.out[i + n * j] = s;
    }
  }
}

void launch_reginv(const RegInvDesc* d_descs, int ndesc, const MFOp* d_ops, int* d_status, cudaStream_t st) {
  if (ndesc <= 0) return;
  // up to four blocks per matrix while the GPU has SMs for them
  const unsigned split = (unsigned)std::max(1, std::min(4, sm_count() / ndesc));
  reginv_kernel<<<dim3(ndesc, split), 128, 0, st>>>(d_descs, d_ops, d_status);
}

// ---------------------------------------------------------------------------
// Natural populations (output.f90:88-140), one warp per (mode, state) block:
// eigenvalues of rho (zheev on the upper triangle) in decreasing order; for a
// Gaussian mode of conj(S^1/2) rho conj(S^1/2) with S^1/2 = sum_j sqrt(w_j) u_j u_j^H
// (SquareRoot, maths.f90:556-585; zlacgv; two zhemm 'R' on upper triangles), the
// gross Gaussian populations sum_j2 Re(rho S)(j1, j2) and the population errors
// |sum_j2 2 Re(rho S)(j1, j2) - rho(j1, j1)| (decreasing), all from upper triangles.
// ---------------------------------------------------------------------------
__device__ __forceinline__ cplx herm_up(const cplx* X, int n, int i, int j) {
  cplx v = (i <= j) ? X[i + n * j] : cconj(X[j + n * i]);
  if (i == j) v.y = 0.0;
  return v;
}

// position of v[i] in decreasing order (ties keep their index order)
__device__ __forceinline__ int rank_desc(const double* v, int n, int i) {
  int r = 0;
  for (int j = 0; j < n; ++j) r += (v[j] > v[i]) || (v[j] == v[i] && j < i);
  return r;
}

__global__ void __launch_bounds__(32) natpop_kernel(const NatpopDesc* __restrict__ descs, int* status) {
  __shared__ cplx A[MAXN_SPF * MAXN_SPF];
  __shared__ cplx V[MAXN_SPF * MAXN_SPF];
  __shared__ double w[MAXN_SPF];
  __shared__ JacRot R[MAXN_SPF / 2];
  const NatpopDesc& d = descs[blockIdx.x];
  const int n = d.n, ld = MAXN_SPF, lane = threadIdx.x;
  bool ok = true, ok2 = true;
  if (d.S) {
    for (int e = lane; e < n * n; e += 32) A[e % n + ld * (e / n)] = herm_up(d.S, n, e % n, e / n);
    __syncwarp();
    jacobi_herm(A, V, n, ld, R, &ok);
    if (lane < n) w[lane] = sqrt(A[lane + ld * lane].x);
    __syncwarp();
    cplx* S12 = d.work;
    cplx* T = d.work + n * n;
    for (int e = lane; e < n * n; e += 32) {
      const int i = e % n, j = e / n;
      cplx v = mkc(0.0, 0.0);
      for (int k = 0; k < n; ++k) v = cadd(v, cscale(cmul(V[i + ld * k], cconj(V[j + ld * k])), w[k]));
      S12[e] = cconj(v);
    }
    __syncwarp();
    for (int e = lane; e < n * n; e += 32) {   // T = S12 rho
      const int i = e % n, j = e / n;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n; ++q) v = cadd(v, cmul(S12[i + n * q], herm_up(d.rho, n, q, j)));
      T[e] = v;
    }
    __syncwarp();
    for (int e = lane; e < n * n; e += 32) {   // M = T S12, S12 Hermitian from its upper triangle
      const int i = e % n, j = e / n;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n; ++q) v = cadd(v, cmul(T[i + n * q], herm_up(S12, n, q, j)));
      A[i + ld * j] = v;
    }
    __syncwarp();
    for (int e = lane; e < n * n; e += 32) {   // zheev reads the upper triangle
      const int i = e % n, j = e / n;
      if (i > j) A[i + ld * j] = cconj(A[j + ld * i]);
      if (i == j) A[i + ld * j].y = 0.0;
    }
  } else {
    for (int e = lane; e < n * n; e += 32) A[e % n + ld * (e / n)] = herm_up(d.rho, n, e % n, e / n);
  }
  __syncwarp();
  jacobi_herm(A, V, n, ld, R, &ok2);
  if (lane < n) w[lane] = A[lane + ld * lane].x;
  __syncwarp();
  if (lane < n) d.natpop[rank_desc(w, n, lane)] = w[lane];
  __syncwarp();
  if (d.S) {
    double g = 0.0, e = 0.0;
    if (lane < n) {
      const int j1 = lane;
      for (int j2 = 0; j2 < j1; ++j2) {
        const double v = cmul(d.rho[j2 + n * j1], d.S[j2 + n * j1]).x;
        g += v;
        e += 2.0 * v;
      }
      e -= d.rho[j1 + n * j1].x;
      for (int j2 = j1; j2 < n; ++j2) {
        const double v = cmul(d.rho[j1 + n * j2], d.S[j1 + n * j2]).x;
        g += v;
        e += 2.0 * v;
      }
      e = fabs(e);
      d.ggp[j1] = g;
      w[lane] = e;
    }
    __syncwarp();
    if (lane < n) d.poperr[rank_desc(w, n, lane)] = e;
  }
  if (lane == 0 && !(ok && ok2)) atomicOr(status, DEVST_EIG_NOCONV);
}
void launch_natpop(const NatpopDesc* d, int nd, int* status, cudaStream_t st) {
  if (nd <= 0) return;
  natpop_kernel<<<nd, 32, 0, st>>>(d, status);
}

// ---------------------------------------------------------------------------
// <a|b> over a whole vector in FP64 (zdotc): each of DOT_BLOCKS blocks sums a
// grid-stride range (warp shuffles, then warps in order), and the last block to
// finish adds the block sums in block order, so the result does not depend on
// the blocks' timing.  The counter is reset for the next launch (graph replays).
// ---------------------------------------------------------------------------
__device__ __forceinline__ cplx warp_sum_c(cplx v) {
  for (int off = 16; off > 0; off >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, off);
    v.y += __shfl_down_sync(0xffffffffu, v.y, off);
  }
  return v;
}

__global__ void __launch_bounds__(256) dot_kernel(const cplx* __restrict__ a, const cplx* __restrict__ b,
                                                  long long n, cplx* partial, unsigned* counter, cplx* out) {
  __shared__ cplx ws[8];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cplx s = mkc(0.0, 0.0);
  for (long long i = (long long)blockIdx.x * blockDim.x + tid; i < n; i += (long long)gridDim.x * blockDim.x) {
    const cplx x = a[i], y = b[i];
    s.x = fma(x.x, y.x, fma(x.y, y.y, s.x));
    s.y = fma(x.x, y.y, fma(-x.y, y.x, s.y));
  }
  s = warp_sum_c(s);
  if (lane == 0) ws[warp] = s;
  __syncthreads();
  if (tid == 0) {
    cplx t = ws[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = cadd(t, ws[w]);
    partial[blockIdx.x] = t;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp == 0) {
    cplx t = mkc(0.0, 0.0);
    for (int q = lane; q < (int)gridDim.x; q += 32) {
      const volatile double* pv = (const volatile double*)partial;
      t = cadd(t, mkc(pv[2 * q], pv[2 * q + 1]));
    }
    t = warp_sum_c(t);
    if (lane == 0) {
      *out = t;
      *counter = 0u;
    }
  }
}
void launch_dot(const cplx* a, const cplx* b, long long n, cplx* partial, unsigned* counter, cplx* out,
                cudaStream_t st) {
  dot_kernel<<<DOT_BLOCKS, 256, 0, st>>>(a, b, n, partial, counter, out);
}

// Tridiagonal eigenproblem of the Lanczos matrix (dstev, cmf2_integration.f90:85), for
// Lanczos runs on FP32 products (see grid_sum_tree).
__global__ void tridiag_kernel(const double* alpha, const double* beta, int n, double* evals, double* evecs,
                               int* status) {
  __shared__ cplx A[MAXN_SPF * MAXN_SPF];
  __shared__ cplx V[MAXN_SPF * MAXN_SPF];
  __shared__ JacRot R[MAXN_SPF / 2];
  const int ld = MAXN_SPF;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    double v = 0.0;
    if (i == j) v = alpha[i];
    else if (j == i + 1) v = beta[i];
    else if (i == j + 1) v = beta[j];
    A[i + ld * j] = mkc(v, 0.0);
  }
  __syncthreads();
  bool ok;
  jacobi_herm(A, V, n, ld, R, &ok);
  if (!ok && threadIdx.x == 0) atomicOr(status, DEVST_EIG_NOCONV);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    evecs[i + n * j] = V[i + ld * j].x;   // real symmetric input keeps V real
  }
  if (threadIdx.x < n) evals[threadIdx.x] = A[threadIdx.x + ld * threadIdx.x].x;
}

void launch_jacobi_tridiag(const double* alpha, const double* beta, int n, double* evals, double* evecs,
                           int* d_status, cudaStream_t st) {
  tridiag_kernel<<<1, 32, 0, st>>>(alpha, beta, n, evals, evecs, d_status);
}

// ---------------------------------------------------------------------------
// Elementwise helpers
// ---------------------------------------------------------------------------
// The launch-wide sum of one complex value per thread, in a fixed order: the block's
// values in shared memory, the components by warps 0 and 1 into partial[blockIdx.x];
// the last block to finish adds the block sums likewise into *out and resets the
// counter (graph replays).  Every thread of every block (256 threads) calls it.  Two
// warps add where a tree in every warp took 85 FP64 instructions per block instead of
// 26.
#define GRID_SUM_THREADS 256
__device__ __forceinline__ void block_sum_c(cplx v, double (*sv)[GRID_SUM_THREADS], cplx* res) {
  const int tid = threadIdx.x, lane = tid & 31;
  sv[0][tid] = v.x;
  sv[1][tid] = v.y;
  __syncthreads();
  if (tid < 64) {
    const double* c = sv[tid >> 5];
    double t = c[lane];
#pragma unroll
    for (int k = 32; k < GRID_SUM_THREADS; k += 32) t += c[lane + k];
    for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
    if (lane == 0) reinterpret_cast<double*>(res)[tid >> 5] = t;
  }
  __syncthreads();
}
__device__ void grid_sum_c(cplx v, cplx* partial, unsigned* counter, cplx* out) {
  __shared__ double sv[2][GRID_SUM_THREADS];
  __shared__ cplx r;
  __shared__ bool last;
  const int tid = threadIdx.x;
  block_sum_c(v, sv, &r);
  if (tid == 0) {
    partial[blockIdx.x] = r;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const volatile double* pv = (const volatile double*)partial;
  cplx t = mkc(0.0, 0.0);
  for (int q = tid; q < (int)gridDim.x; q += GRID_SUM_THREADS) t = cadd(t, mkc(pv[2 * q], pv[2 * q + 1]));
  block_sum_c(t, sv, &r);
  if (tid == 0) {
    *out = r;
    *counter = 0u;
  }
}

// The same with a tree in every warp, the order of Lanczos runs on FP32 products: these
// round every Krylov vector to FP32, so that a last-bit change of a sum (or of the
// eigenvectors above) is carried to FP32 level within a few steps; these runs keep one
// arithmetic, which costs about 300 us a CMF2 step of the 8-SPF QVC model.
__device__ __forceinline__ cplx warp_sum_cd(cplx v) {
  for (int off = 16; off > 0; off >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, off);
    v.y += __shfl_down_sync(0xffffffffu, v.y, off);
  }
  return v;
}
__device__ void grid_sum_tree(cplx v, cplx* partial, unsigned* counter, cplx* out) {
  __shared__ cplx ws[32];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum_cd(v);
  if (lane == 0) ws[warp] = v;
  __syncthreads();
  if (tid == 0) {
    cplx t = ws[0];
    for (int w = 1; w < nw; ++w) t = cadd(t, ws[w]);
    partial[blockIdx.x] = t;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const volatile double* pv = (const volatile double*)partial;
  cplx t = mkc(0.0, 0.0);
  for (int q = tid; q < (int)gridDim.x; q += blockDim.x) t = cadd(t, mkc(pv[2 * q], pv[2 * q + 1]));
  t = warp_sum_cd(t);
  __syncthreads();
  if (lane == 0) ws[warp] = t;
  __syncthreads();
  if (tid == 0) {
    cplx r = ws[0];
    for (int w = 1; w < nw; ++w) r = cadd(r, ws[w]);
    *out = r;
    *counter = 0u;
  }
}

// out[i] = sum_k coeff_k src_k[i - offset] over the sources of the state range
// holding i; with dot.v also the launch-wide <dot.v|out> (FP64 products of the
// values written) into dot.res.  The warps of the launch take rows of 32 elements in
// turn: contiguous shares per block left every thread a sixth, nearly empty round at
// 786,432 elements.
// PREC 0: FP64, bound by its instructions: two per source with a real or an imaginary
// coefficient (every term of a Hamiltonian with real coefficients), four otherwise.
// The sources come sorted by kind; told apart inside the loop they were issued under
// predicates and all paid for (8-SPF QVC model, about ten sources a state: 107 -> 51 us with the inner product, 48 -> 43 without).
// PREC 1: FP32 coefficients times FP32-rounded sources accumulated in FP32 (the
// sources are FP32 products there); two elements per thread, bound by the loads in flight
// (8-SPF QVC model, about ten sources a state: 39 -> 28 us).
#define TERMSUM_CACHE 64
// KIND 0 complex, 1 imaginary, 2 real
template <int KIND>
__device__ __forceinline__ void termsum_run(cplx& val, const SumSrc* sp, int n, long long li) {
  for (int k0 = 0; k0 < n; k0 += 4) {
    cplx x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k0 + k < n) x[k] = load_c(sp[k0 + k].src, li, sp[k0 + k].fmt);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k0 + k >= n) break;
      const cplx c = sp[k0 + k].coeff;
      if (KIND == 1) {
        val.x = fma(-c.y, x[k].y, val.x);
        val.y = fma(c.y, x[k].x, val.y);
      } else if (KIND == 2) {
        val.x = fma(c.x, x[k].x, val.x);
        val.y = fma(c.x, x[k].y, val.y);
      } else {
        cfma(val, c, x[k]);
      }
    }
  }
}
// FP32: N (1 or 2) neighbouring elements from li on into a (re, im each)
template <int N>
__device__ __forceinline__ void termsum_f32(float* a, const SumSrc* sp, int n, long long li) {
  for (int k0 = 0; k0 < n; k0 += 4) {
    float4 x[4][N];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k0 + k < n) {
        const SumSrc& s = sp[k0 + k];
        if (N == 2 && s.fmt) {   // 16 bytes hold both
          const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float2*>(s.src) + li);
          x[k][0] = make_float4(v.x, v.y, 0.f, 0.f);
          x[k][N - 1] = make_float4(v.z, v.w, 0.f, 0.f);
        } else {
#pragma unroll
          for (int e = 0; e < N; ++e) x[k][e] = load_split(s.src, li + e, s.fmt);
        }
      }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k0 + k >= n) break;
      const float cr = sp[k0 + k].cs[0] + sp[k0 + k].cs[1], ci = sp[k0 + k].cs[2] + sp[k0 + k].cs[3];
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const float xr = x[k][e].x + x[k][e].z, xi = x[k][e].y + x[k][e].w;
        a[2 * e] = fmaf(cr, xr, fmaf(-ci, xi, a[2 * e]));
        a[2 * e + 1] = fmaf(cr, xi, fmaf(ci, xr, a[2 * e + 1]));
      }
    }
  }
}
template <int PREC>
__global__ void __launch_bounds__(256, 4) termsum_kernel(cplx* __restrict__ out, const SumRange* __restrict__ ranges,
                                                      int nr, const SumSrc* __restrict__ srcs, long long total,
                                                      FusedDot dot) {
  __shared__ SumSrc ss[TERMSUM_CACHE];
  const int nsrc = ranges[nr - 1].first + ranges[nr - 1].count;
  const bool cached = nsrc <= TERMSUM_CACHE;
  if (cached)
    for (int k = threadIdx.x; k < nsrc; k += blockDim.x) ss[k] = srcs[k];
  __syncthreads();
  const SumSrc* all = cached ? ss : srcs;
  cplx d = mkc(0, 0);
  SumRange rg;
  rg.offset = rg.n = 0;
  // warp w of the launch: neighbouring warps of a block work far apart
  constexpr int N = PREC == 1 ? 2 : 1;   // elements per thread and row
  const long long wrow = ((long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
  const long long stride = (long long)N * gridDim.x * blockDim.x;
  for (long long i0 = N * wrow, i = i0; i < total; i = i + 1 < min(total, i0 + N) ? i + 1 : (i0 += stride)) {
    if (i - rg.offset >= rg.n) {
      int lo = 0, hi = nr - 1;   // last range starting at or before i (ranges sorted by offset)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ranges[mid].offset <= i) lo = mid; else hi = mid - 1;
      }
      rg = ranges[lo];
      if (i - rg.offset >= rg.n || i < rg.offset) {   // outside every range
        rg.n = 0;
        continue;
      }
    }
    const long long li = i - rg.offset;
    const SumSrc* sp = all + rg.first;
    // both of a pair: the FP32 sources are whole allocations, 16-byte aligned at even li
    if (PREC == 1 && i == i0 && !(li & 1) && li + 1 < rg.n) {
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      termsum_f32<2>(a, sp, rg.count, li);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const cplx v = mkc(f2d_exact(a[2 * e]), f2d_exact(a[2 * e + 1]));
        out[i + e] = v;
        if (dot.v) cfma_conj(d, dot.v[i + e], v);
      }
      ++i;
      continue;
    }
    cplx val;
    if (PREC == 1) {
      float a[2] = {0.f, 0.f};
      termsum_f32<1>(a, sp, rg.count, li);
      val = mkc(f2d_exact(a[0]), f2d_exact(a[1]));
    } else {
      val = mkc(0, 0);
      termsum_run<1>(val, sp, rg.nimag, li);
      termsum_run<2>(val, sp + rg.nimag, rg.nreal, li);
      termsum_run<0>(val, sp + rg.nimag + rg.nreal, rg.count - rg.nimag - rg.nreal, li);
    }
    out[i] = val;
    if (dot.v) cfma_conj(d, dot.v[i], val);
  }
  if (dot.v) grid_sum_c(d, dot.partial, dot.counter, dot.res);
}

// FP32 term sum with the launch-wide <dot.v|out> in the order of grid_sum_tree: contiguous
// shares per block, four elements per thread in flight.
__global__ void __launch_bounds__(256) termsum_f32_dot_kernel(cplx* __restrict__ out, const SumRange* __restrict__ ranges,
                                                      int nr, const SumSrc* __restrict__ srcs, long long total,
                                                      FusedDot dot) {
  __shared__ SumSrc ss[TERMSUM_CACHE];
  __shared__ int s_rg;
  const long long chunk = (total + gridDim.x - 1) / gridDim.x;
  const long long start = (long long)blockIdx.x * chunk, end = min(total, start + chunk);
  cplx d = mkc(0, 0);
  long long base = start;
  while (base < end) {
    if (threadIdx.x == 0) {
      int lo = 0, hi = nr - 1;   // last range starting at or before base (ranges sorted by offset)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ranges[mid].offset <= base) lo = mid; else hi = mid - 1;
      }
      s_rg = lo;
    }
    __syncthreads();
    const SumRange rg = ranges[s_rg];
    long long seg_end = min(end, rg.offset + rg.n);
    if (base < rg.offset || base >= rg.offset + rg.n) {
      // outside every range: skip to the next range start
      seg_end = (s_rg + 1 < nr) ? min(end, ranges[s_rg + 1].offset) : end;
      __syncthreads();
      base = max(seg_end, base + 1);
      continue;
    }
    const bool cached = rg.count <= TERMSUM_CACHE;
    if (cached)
      for (int k = threadIdx.x; k < rg.count; k += blockDim.x) ss[k] = srcs[rg.first + k];
    __syncthreads();
    const SumSrc* sp = cached ? ss : srcs + rg.first;
    {
      // four elements per thread in flight: per source, four independent loads
      const long long stride = (long long)blockDim.x;
      for (long long i0 = base + threadIdx.x; i0 < seg_end; i0 += 4 * stride) {
        float ar[4] = {0.f, 0.f, 0.f, 0.f}, ai[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < rg.count; ++k) {
          const float cr = sp[k].cs[0] + sp[k].cs[1], ci = sp[k].cs[2] + sp[k].cs[3];
          const cplx* src = sp[k].src;
          const int fmt = sp[k].fmt;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const long long i = i0 + e * stride;
            if (i >= seg_end) break;
            const float4 x = load_split(src, i - rg.offset, fmt);
            const float xr = x.x + x.z, xi = x.y + x.w;
            ar[e] = fmaf(cr, xr, fmaf(-ci, xi, ar[e]));
            ai[e] = fmaf(cr, xi, fmaf(ci, xr, ai[e]));
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const long long i = i0 + e * stride;
          if (i >= seg_end) break;
          const cplx val = mkc(f2d_exact(ar[e]), f2d_exact(ai[e]));
          out[i] = val;
          cfma_conj(d, dot.v[i], val);
        }
      }
      __syncthreads();
      base = seg_end;
    }
  }
  grid_sum_tree(d, dot.partial, dot.counter, dot.res);
}

void launch_termsum(cplx* out, const SumRange* d_ranges, int nranges, const SumSrc* d_srcs, long long total,
                    cudaStream_t st, int prec, FusedDot dot) {
  if (total <= 0) return;
  const unsigned nb = (unsigned)std::min<long long>((total + 255) / 256, FUSED_BLOCKS);
  if (prec == 1 && dot.v)
    termsum_f32_dot_kernel<<<nb, 256, 0, st>>>(out, d_ranges, nranges, d_srcs, total, dot);
  else if (prec == 1)
    termsum_kernel<1><<<nb, 256, 0, st>>>(out, d_ranges, nranges, d_srcs, total, dot);
  else
    termsum_kernel<0><<<nb, 256, 0, st>>>(out, d_ranges, nranges, d_srcs, total, dot);
}

__global__ void stage_kernel(cplx* __restrict__ out, const cplx* __restrict__ base, StageArgs a, double dt,
                             long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  cplx s = mkc(0, 0);
  for (int k = 0; k < a.nk; ++k) {
    cplx v = a.k[k][i];
    s.x = fma(a.c[k], v.x, s.x);
    s.y = fma(a.c[k], v.y, s.y);
  }
  cplx b = base[i];
  out[i] = mkc(fma(dt, s.x, b.x), fma(dt, s.y, b.y));
}

// Ensemble stage: every member m (elements off[m] .. off[m+1]) with its own dt.
__device__ __forceinline__ int member_of(const long long* __restrict__ off, int nm, long long i) {
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}
__global__ void ens_stage_kernel(cplx* __restrict__ out, const cplx* __restrict__ base, StageArgs a,
                                 const double* __restrict__ dt, const long long* __restrict__ off, int nm,
                                 long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double h = dt[member_of(off, nm, i)];
  cplx s = mkc(0, 0);
  for (int k = 0; k < a.nk; ++k) {
    cplx v = a.k[k][i];
    s.x = fma(a.c[k], v.x, s.x);
    s.y = fma(a.c[k], v.y, s.y);
  }
  cplx b = base[i];
  out[i] = mkc(fma(h, s.x, b.x), fma(h, s.y, b.y));
}
void launch_ens_stage(cplx* out, const cplx* base, const StageArgs& a, const double* dt, const long long* off, int nm,
                      long long n, cudaStream_t st) {
  if (n <= 0) return;
  ens_stage_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, base, a, dt, off, nm, n);
}
__global__ void ens_accept_kernel(cplx* __restrict__ y, const cplx* __restrict__ src, const int* __restrict__ accept,
                                  const long long* __restrict__ off, int nm, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (accept[member_of(off, nm, i)]) y[i] = src[i];
}
void launch_ens_accept(cplx* y, const cplx* src, const int* accept, const long long* off, int nm, long long n,
                       cudaStream_t st) {
  if (n <= 0) return;
  ens_accept_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y, src, accept, off, nm, n);
}

__global__ void bs_final_kernel(cplx* __restrict__ out, const cplx* __restrict__ am, const cplx* __restrict__ an,
                                const cplx* __restrict__ d, double dt, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const cplx a = am[i], b = an[i], g = d[i];
  out[i] = mkc(0.5 * ((a.x + b.x) + dt * g.x), 0.5 * ((a.y + b.y) + dt * g.y));
}
void launch_bs_final(cplx* out, const cplx* am, const cplx* an, const cplx* d, double dt, long long n, cudaStream_t st) {
  if (n <= 0) return;
  bs_final_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, am, an, d, dt, n);
}
__global__ void bs_extr_kernel(BsExtr e, const cplx* __restrict__ est, cplx* __restrict__ a0, cplx* __restrict__ a1,
                               long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const cplx x = est[i];
  if (e.iest == 1) {
    e.q[1][i] = x;
    a0[i] = x;
    a1[i] = x;
    return;
  }
  cplx A0 = x, A1 = x, At = x;
  for (int k1 = 1; k1 < e.iest; ++k1) {
    const cplx cd = e.q[k1][i];
    e.q[k1][i] = A1;
    const cplx del = csub(At, cd);
    A1 = cscale(del, e.f1[k1]);
    At = cscale(del, e.f2[k1]);
    A0 = cadd(A0, A1);
  }
  e.q[e.iest][i] = A1;
  a0[i] = A0;
  a1[i] = cadd(A0, A1);
}
void launch_bs_extr(const BsExtr& e, const cplx* est, cplx* a0, cplx* a1, long long n, cudaStream_t st) {
  if (n <= 0) return;
  bs_extr_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(e, est, a0, a1, n);
}

void launch_stage(cplx* out, const cplx* base, const StageArgs& a, double dt, long long n, cudaStream_t st) {
  if (n <= 0) return;
  stage_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, base, a, dt, n);
}

__global__ void copy_scale_kernel(cplx* out, const cplx* in, cplx s, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = cmul(s, in[i]);
}
void launch_copy_scale(cplx* out, const cplx* in, cplx s, long long n, cudaStream_t st) {
  if (n <= 0) return;
  copy_scale_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, in, s, n);
}

__global__ void axpy_kernel(cplx* y, const cplx* x, cplx a, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { cplx v = y[i]; cfma(v, a, x[i]); y[i] = v; }
}
// complex FP64 -> complex FP32 rounded to nearest (the FP64 pipe stays idle)
__global__ void to_f32_kernel(float2* __restrict__ out, const cplx* __restrict__ in, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const cplx v = in[i];
  float hx, lx, hy, ly;
  split_d2f(v.x, hx, lx);
  split_d2f(v.y, hy, ly);
  out[i] = make_float2(hx + lx, hy + ly);
}
void launch_to_f32(cplx* out, const cplx* in, long long n, cudaStream_t st) {
  if (n <= 0) return;
  to_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(reinterpret_cast<float2*>(out), in, n);
}

void launch_axpy(cplx* y, const cplx* x, cplx a, long long n, cudaStream_t st) {
  if (n <= 0) return;
  axpy_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y, x, a, n);
}

// out = sum_j coef_j basis_j, and with nrm.res the launch-wide ||out||^2
__global__ void __launch_bounds__(256) gemv_cols_kernel(cplx* __restrict__ out, const cplx* __restrict__ basis,
                                                        long long ld, const cplx* __restrict__ coef, int ncol,
                                                        long long n, FusedDot nrm) {
  double s2 = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    cplx s = mkc(0, 0);
#pragma unroll 4
    for (int j = 0; j < ncol; ++j) cfma(s, coef[j], basis[i + ld * j]);
    out[i] = s;
    s2 = fma(s.x, s.x, fma(s.y, s.y, s2));
  }
  if (nrm.res) grid_sum_c(mkc(s2, 0.0), nrm.partial, nrm.counter, nrm.res);
}
void launch_gemv_cols(cplx* out, const cplx* basis, long long ld, const cplx* coef, int ncol, long long n,
                      cudaStream_t st, FusedDot nrm) {
  const unsigned nb = (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, FUSED_BLOCKS));
  gemv_cols_kernel<<<nb, 256, 0, st>>>(out, basis, ld, coef, ncol, n, nrm);
}

// ---------------------------------------------------------------------------
// FP64 FMA throughput calibration (independent FMA chains, no memory traffic).
// ---------------------------------------------------------------------------
__global__ void fp64_peak_kernel(double* out, int iters, double a) {
  double x0 = threadIdx.x * 1e-3, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
         x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, 1e-9); x1 = fma(x1, a, 1e-9); x2 = fma(x2, a, 1e-9); x3 = fma(x3, a, 1e-9);
    x4 = fma(x4, a, 1e-9); x5 = fma(x5, a, 1e-9); x6 = fma(x6, a, 1e-9); x7 = fma(x7, a, 1e-9);
  }
  double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == 12345.678) out[0] = s;
}

double measure_fp64_tflops() {
  double* d = nullptr;
  if (cudaMalloc(&d, 64) != cudaSuccess) return 0.0;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = nsm * 8, threads = 256, iters = 4096;
  fp64_peak_kernel<<<blocks, threads>>>(d, 16, 0.999999);
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    cudaEventRecord(a);
    fp64_peak_kernel<<<blocks, threads>>>(d, iters, 0.999999);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms;
    cudaEventElapsedTime(&ms, a, b);
    best = ms < best ? ms : best;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(d);
  const double flops = 2.0 * 8.0 * (double)iters * blocks * threads;
  return flops / (best * 1e-3) / 1e12;
}

// ---------------------------------------------------------------------------
// Lockstep SPF integration of all DVR modes (rk_SPF_ck with frozen mean fields,
// cmf2_integration.f90:105-253): every psi element carries its mode, each mode its
// own step length (0 for a mode that has finished its interval).
// ---------------------------------------------------------------------------
__global__ void stage_modes_kernel(cplx* __restrict__ out, const cplx* __restrict__ base, StageArgs a,
                                   const double* __restrict__ dt_mode, const unsigned char* __restrict__ elem_mode,
                                   long long off, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long g = off + i;
  const double dt = dt_mode[elem_mode[i]];
  cplx s = mkc(0, 0);
  for (int k = 0; k < a.nk; ++k) {
    cplx v = a.k[k][g];
    s.x = fma(a.c[k], v.x, s.x);
    s.y = fma(a.c[k], v.y, s.y);
  }
  cplx b = base[g];
  out[g] = mkc(fma(dt, s.x, b.x), fma(dt, s.y, b.y));
}
void launch_stage_modes(cplx* out, const cplx* base, const StageArgs& a, const double* dt_mode,
                        const unsigned char* elem_mode, long long off, long long n, cudaStream_t st) {
  if (n <= 0) return;
  stage_modes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, base, a, dt_mode, elem_mode, off, n);
}

__global__ void rk_end_kernel(cplx* __restrict__ y5, cplx* __restrict__ diff, const cplx* __restrict__ base, StageArgs a,
                              StageArgs a4, const double* __restrict__ dt_mode,
                              const unsigned char* __restrict__ elem_mode, long long off, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long g = off + i;
  const double dt = dt_mode[elem_mode[i]];
  cplx s = mkc(0, 0), r = mkc(0, 0);
  for (int k = 0; k < a.nk; ++k) {
    const cplx v = a.k[k][g];
    s.x = fma(a.c[k], v.x, s.x);
    s.y = fma(a.c[k], v.y, s.y);
    r.x = fma(a4.c[k], v.x, r.x);
    r.y = fma(a4.c[k], v.y, r.y);
  }
  const cplx b = base[g];
  const cplx u = mkc(fma(dt, s.x, b.x), fma(dt, s.y, b.y)), w = mkc(fma(dt, r.x, b.x), fma(dt, r.y, b.y));
  y5[g] = u;
  diff[g] = csub(u, w);
}
void launch_rk_end(cplx* y5, cplx* diff, const cplx* base, const StageArgs& a, const double* c4, const double* dt_mode,
                   const unsigned char* elem_mode, long long off, long long n, cudaStream_t st) {
  if (n <= 0) return;
  StageArgs a4 = a;
  for (int k = 0; k < a.nk; ++k) a4.c[k] = c4[k];
  rk_end_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y5, diff, base, a, a4, dt_mode, elem_mode, off, n);
}

// y <- src on the elements of accepted modes
__global__ void masked_copy_kernel(cplx* __restrict__ y, const cplx* __restrict__ src,
                                   const unsigned char* __restrict__ elem_mode, const int* __restrict__ accept,
                                   long long off, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (accept[elem_mode[i]]) y[off + i] = src[off + i];
}
void launch_masked_copy(cplx* y, const cplx* src, const unsigned char* elem_mode, const int* accept, long long off,
                        long long n, cudaStream_t st) {
  if (n <= 0) return;
  masked_copy_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(y, src, elem_mode, accept, off, n);
}

// Calc_Err_SPF (cmf2_derivatives.f90:239-283): err_m = sqrt|sum_blocks Tr(rho dS)| with
// the reference's upper-triangle evaluation; one thread per mode.
// err_m = sqrt|sum over the mode's blocks of Tr(rho . dS)| (Calc_Err_SPF,
// cmf2_derivatives.f90:239-338): one warp per block (lane-strided entries,
// shuffle sum), then one thread per mode adds its blocks in descriptor order.
__global__ void __launch_bounds__(1024) spf_err_kernel(const SpfErrDesc* __restrict__ d, int nd, double* err_mode,
                                                       int nmodes) {
  __shared__ double part[256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5;
  for (int q = warp; q < nd && q < 256; q += nw) {
    const int n = d[q].n;
    const cplx* r = d[q].rho;
    const cplx* o = d[q].ds;
    double e = 0.0;
    for (int pr = lane; pr < n * n; pr += 32) {
      const int j1 = pr % n, j2 = pr / n;
      if (j1 > j2) continue;
      const cplx rv = r[pr], ov = o[pr];
      e += (j1 < j2) ? 2.0 * (rv.x * ov.x + rv.y * ov.y) : (rv.x * ov.x - rv.y * ov.y);
    }
    for (int off = 16; off > 0; off >>= 1) e += __shfl_down_sync(0xffffffffu, e, off);
    if (lane == 0) part[q] = e;
  }
  __syncthreads();
  const int m = threadIdx.x;
  if (m >= nmodes) return;
  double e = 0.0;
  bool any = false;
  for (int q = 0; q < nd && q < 256; ++q) {
    if (d[q].mode != m) continue;
    any = true;
    e += part[q];
  }
  err_mode[m] = any ? sqrt(fabs(e)) : 0.0;
}
void launch_spf_err(const SpfErrDesc* d, int nd, double* err_mode, int nmodes, cudaStream_t st) {
  // nd <= 256 blocks (checked when the plan is built), nmodes <= 64
  const int warps = std::max(std::min(nd, 32), (nmodes + 31) / 32);
  spf_err_kernel<<<1, 32 * warps, 0, st>>>(d, nd, err_mode, nmodes);
}

// ---------------------------------------------------------------------------
// Lanczos recurrence with device-resident scalars (cmf2_integration.f90:53-79):
// Kn <- (Kn - beta_prev * Kp) - alpha * Kj, alpha = Re <Kj|Kn> (two zaxpy in the
// reference order), then Kn <- Kn / ||Kn||.
// ---------------------------------------------------------------------------
// ... and with nrm.res the launch-wide ||Kn||^2 of the new Kn (the next normalisation)
__global__ void lan_axpy_kernel(cplx* __restrict__ Kn, const cplx* __restrict__ Kj, const cplx* __restrict__ Kp,
                                const cplx* __restrict__ dot_alpha, const double* __restrict__ beta_prev,
                                double* alpha_out, long long n, FusedDot nrm) {
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const double alpha = dot_alpha->x;
  if (i0 == 0) *alpha_out = alpha;
  const double b = Kp ? *beta_prev : 0.0;
  double s2 = 0.0;
  for (long long i = i0; i < n; i += (long long)gridDim.x * blockDim.x) {
    cplx v = Kn[i];
    if (Kp) {
      cplx p = Kp[i];
      v = mkc(fma(-b, p.x, v.x), fma(-b, p.y, v.y));
    }
    cplx q = Kj[i];
    const cplx w = mkc(fma(-alpha, q.x, v.x), fma(-alpha, q.y, v.y));
    Kn[i] = w;
    s2 = fma(w.x, w.x, fma(w.y, w.y, s2));
  }
  if (nrm.res) grid_sum_tree(mkc(s2, 0.0), nrm.partial, nrm.counter, nrm.res);
}
void launch_lan_axpy(cplx* Kn, const cplx* Kj, const cplx* Kp, const cplx* dot_alpha, const double* beta_prev,
                     double* alpha_out, long long n, cudaStream_t st, FusedDot nrm) {
  const unsigned nb = (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, FUSED_BLOCKS));
  lan_axpy_kernel<<<nb, 256, 0, st>>>(Kn, Kj, Kp, dot_alpha, beta_prev, alpha_out, n, nrm);
}

// Grid-stride: the norm and its reciprocal once per block (an FP64 square root and a
// division take 1,160 cycles of a sub-partition's FP64 pipe per warp), then one multiply
// per component.
// ... optionally also into copy (FP64) and f32 (complex FP32 rounded to nearest):
// the input of the next H_B application, written in the same pass.
__global__ void lan_normalize_kernel(cplx* __restrict__ out, const cplx* __restrict__ in, const cplx* __restrict__ nrm2,
                                     double* beta_out, long long n, cplx* __restrict__ copy,
                                     float2* __restrict__ f32) {
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ double s_inv;
  if (threadIdx.x == 0) {
    const double beta = sqrt(nrm2->x);
    if (blockIdx.x == 0 && beta_out) *beta_out = beta;
    s_inv = 1.0 / beta;
  }
  __syncthreads();
  const double s = s_inv;
  for (long long i = i0; i < n; i += (long long)gridDim.x * blockDim.x) {
    const cplx v = in[i];
    const cplx w = mkc(v.x * s, v.y * s);
    out[i] = w;
    if (copy) copy[i] = w;
    if (f32) {
      float hx, lx, hy, ly;
      split_d2f(w.x, hx, lx);
      split_d2f(w.y, hy, ly);
      f32[i] = make_float2(hx + lx, hy + ly);
    }
  }
}
void launch_lan_normalize(cplx* out, const cplx* in, const cplx* nrm2, double* beta_out, long long n, cudaStream_t st,
                          cplx* copy, cplx* f32) {
  const long long want = (n + 255) / 256;
  const unsigned nb = (unsigned)std::max<long long>(1, std::min<long long>(want, 4LL * sm_count()));
  lan_normalize_kernel<<<nb, 256, 0, st>>>(out, in, nrm2, beta_out, n, copy, reinterpret_cast<float2*>(f32));
}

// ---------------------------------------------------------------------------
// Mean-field snapshots for the learned extrapolator: all density matrices and
// mean fields of the grid modes gathered into one complex vector (and back;
// scatter 2: the mean fields only).
// ---------------------------------------------------------------------------
__global__ void snap_gather_kernel(const SnapSeg* __restrict__ segs, int nseg, cplx* __restrict__ flat, long long E,
                                   int scatter) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E) return;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (segs[mid].offset <= i) lo = mid; else hi = mid - 1;
  }
  cplx* p = segs[lo].ptr + (i - segs[lo].offset);
  if (scatter == 2 && segs[lo].density) return;
  if (scatter) *p = flat[i]; else flat[i] = *p;
}
void launch_snap(const SnapSeg* segs, int nseg, cplx* flat, long long E, int scatter, cudaStream_t st) {
  if (E <= 0) return;
  snap_gather_kernel<<<(unsigned)((E + 255) / 256), 256, 0, st>>>(segs, nseg, flat, E, scatter);
}

// Learned mean-field extrapolation.  Each entry z of the snapshot has its values
// z_0..z_4 at the last five step starts.  Newton increments at tau:
// inc_o(tau) = P_o(tau) - P_{o-1}(tau), P_o the Lagrange polynomial through the
// last o+1 values (P_0 = z_4), with host-computed weights c.inc[tau][o-1][j].
// The scale S is the RMS over all entries of |inc_1| at the step end.

// S = sqrt(mean |inc_1(end)|^2): one block, fixed-order grid-stride sums.
__global__ void __launch_bounds__(1024) mfx_scale_kernel(MfxHist hz, MfxCoef c, double* __restrict__ S,
                                                         long long E) {
  __shared__ double red[1024];
  double acc = 0.0;
  for (long long i = threadIdx.x; i < E; i += blockDim.x) {
    cplx v = mkc(0, 0);
#pragma unroll
    for (int j = 0; j < MFX_NHIST; ++j) {
      const cplx z = hz.z[j][i];
      v.x += c.inc[1][0][j] * z.x;
      v.y += c.inc[1][0][j] * z.y;
    }
    acc += cabs2(v);
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) S[0] = fmax(sqrt(red[0] / (double)(E > 0 ? E : 1)), 1e-300);
}

// The entry's own scale: |inc_1| + |inc_2| at the step end plus 1e-12 S.
__device__ __forceinline__ double mfx_entry_scale(const cplx* z, const MfxCoef& c, double S) {
  cplx v1 = mkc(0, 0), v2 = mkc(0, 0);
#pragma unroll
  for (int j = 0; j < MFX_NHIST; ++j) {
    v1.x += c.inc[1][0][j] * z[j].x;
    v1.y += c.inc[1][0][j] * z[j].y;
    v2.x += c.inc[1][1][j] * z[j].x;
    v2.y += c.inc[1][1][j] * z[j].y;
  }
  return sqrt(cabs2(v1)) + sqrt(cabs2(v2)) + 1e-12 * S + 1e-300;
}

// Network inputs per entry: Re/Im of inc_1..inc_4 at the half step and the step
// end divided by the entry's scale, then the step-length ratios; each divided by
// its column scale.
__global__ void mfx_features_kernel(MfxHist hz, MfxCoef c, const double* __restrict__ S, float* __restrict__ X,
                                    long long E) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E) return;
  cplx z[MFX_NHIST];
#pragma unroll
  for (int j = 0; j < MFX_NHIST; ++j) z[j] = hz.z[j][i];
  const double q = 1.0 / mfx_entry_scale(z, c, S[0]);
  float* x = X + (long long)MFX_NFEAT * i;
  int col = 0;
#pragma unroll
  for (int tau = 0; tau < 2; ++tau) {
#pragma unroll
    for (int o = 0; o < MFX_NHIST - 1; ++o) {
      cplx v = mkc(0, 0);
#pragma unroll
      for (int j = 0; j < MFX_NHIST; ++j) {
        v.x += c.inc[tau][o][j] * z[j].x;
        v.y += c.inc[tau][o][j] * z[j].y;
      }
      x[col] = (float)(v.x * q / c.fscale[col]);
      ++col;
      x[col] = (float)(v.y * q / c.fscale[col]);
      ++col;
    }
  }
#pragma unroll
  for (int r = 0; r < MFX_NHIST - 1; ++r, ++col) x[col] = (float)(c.ratio[r] / c.fscale[col]);
}

// z(tau) = polynomial extrapolation + s * tscale * y at the half step and the step
// end (s the entry's scale)
__global__ void mfx_combine_kernel(MfxHist hz, MfxCoef c, const float* __restrict__ Y, const double* __restrict__ S,
                                   cplx* __restrict__ half, cplx* __restrict__ full, long long E) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E) return;
  cplx z[MFX_NHIST];
#pragma unroll
  for (int j = 0; j < MFX_NHIST; ++j) z[j] = hz.z[j][i];
  const float* y = Y + (long long)MFX_NOUT * i;
  const double s = mfx_entry_scale(z, c, S[0]);
  cplx out[2];
#pragma unroll
  for (int tau = 0; tau < 2; ++tau) {
    cplx v = mkc(0, 0);
#pragma unroll
    for (int j = 0; j < MFX_NHIST; ++j) {
      v.x += c.base[tau][j] * z[j].x;
      v.y += c.base[tau][j] * z[j].y;
    }
    v.x += s * c.tscale[2 * tau] * (double)y[2 * tau];
    v.y += s * c.tscale[2 * tau + 1] * (double)y[2 * tau + 1];
    out[tau] = v;
  }
  half[i] = out[0];
  full[i] = out[1];
}

void launch_mfx_features(const MfxHist& hz, const MfxCoef& c, double* S, float* X, long long E, cudaStream_t st) {
  if (E <= 0) return;
  mfx_scale_kernel<<<1, 1024, 0, st>>>(hz, c, S, E);
  mfx_features_kernel<<<(unsigned)((E + 255) / 256), 256, 0, st>>>(hz, c, S, X, E);
}
void launch_mfx_combine(const MfxHist& hz, const MfxCoef& c, const float* Y, const double* S, cplx* half, cplx* full,
                        long long E, cudaStream_t st) {
  if (E <= 0) return;
  mfx_combine_kernel<<<(unsigned)((E + 255) / 256), 256, 0, st>>>(hz, c, Y, S, half, full, E);
}

// ---------------------------------------------------------------------------
// Statistical mixtures and dissipation
// ---------------------------------------------------------------------------

// Partial sums of <X_i|Y_j> (one row of PK_GRAM_BLOCKS blocks per pair).
__global__ void __launch_bounds__(256) pk_gram_kernel(const PkGramPair* __restrict__ pairs,
                                                      const PkState* __restrict__ st, int nstates,
                                                      cplx* __restrict__ partial) {
  const PkGramPair pr = pairs[blockIdx.y];
  double re = 0.0, im = 0.0;
  for (int s = 0; s < nstates; ++s) {
    const PkState q = st[s];
    const cplx* x = pr.X + q.off + (long long)pr.i * q.n;
    const cplx* y = pr.Y + q.off + (long long)pr.j * q.n;
    for (long long c = blockIdx.x * 256LL + threadIdx.x; c < q.n; c += 256LL * gridDim.x) {
      const cplx a = x[c], b = y[c];
      re = fma(a.x, b.x, fma(a.y, b.y, re));
      im = fma(a.x, b.y, fma(-a.y, b.x, im));
    }
  }
  __shared__ double sr[8], si[8];
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sr[w] = re; si[w] = im; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0, i2 = 0.0;
    for (int k = 0; k < 8; ++k) { r += sr[k]; i2 += si[k]; }
    partial[(long long)blockIdx.y * PK_GRAM_BLOCKS + blockIdx.x] = make_double2(r, i2);
  }
}

void launch_pk_gram(const PkGramPair* d_pairs, int npairs, const PkState* d_st, int nstates, cplx* partial,
                    cudaStream_t st) {
  if (npairs <= 0) return;
  pk_gram_kernel<<<dim3(PK_GRAM_BLOCKS, npairs), 256, 0, st>>>(d_pairs, d_st, nstates, partial);
}

__device__ __forceinline__ cplx pk_mul(cplx a, cplx b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ cplx pk_conj(cplx a) { return make_double2(a.x, -a.y); }

// Packet populations, Lagrange multipliers and mixing matrices (one block).
// WPpopm1 = p / (p^2 + (eps exp(-(p/eps)^2))^2) (gmctdh_objects.f90:616-619);
// type 1 (:661-692): AVA = <A_i|V A_j>, multLagDiag -= aeD1 sum |AVA_ij|^2 WPpopm1_i,
// multLag_ij += aeD1 (AVA AVA^H)_ij (WPpopm1_i + WPpopm1_j) for i > j, D_W += aeD1 WPpopm1_W
// sum_j V A_j conj(AVA_Wj), AuxA_W = i aeD1 WPpopm1_W sum_j A_j conj(AVA_Wj);
// type 2 (:805-818) with G_ij = <A_i|X A_j>, X = sum_t f i aeD2 ae_t W_t:
// multLagDiag -= Re sum_W G_WW, multLag_ij += G_ij + conj(G_ji) for i > j;
// then multLag_ij *= i dw / (dw^2 + (eps exp(-(dw/eps)^2))^2), dw = p_i - p_j (:1128-1137).
__global__ void __launch_bounds__(256) pk_coef_kernel(PkCoefArgs a) {
  extern __shared__ cplx g[];   // [npairs]
  __shared__ double pop[MAX_PACKETS], wpm1[MAX_PACKETS];
  __shared__ cplx M[MAX_PACKETS * MAX_PACKETS];
  __shared__ double dterm[MAX_PACKETS * MAX_PACKETS];
  // one warp per pair: the PK_GRAM_BLOCKS (= 32) block sums, one per lane, added by
  // a fixed shuffle tree
  const int lane = threadIdx.x & 31, tid = threadIdx.x;
  for (int p = tid >> 5; p < a.npairs; p += blockDim.x >> 5) {
    const cplx v = a.partial[(long long)p * PK_GRAM_BLOCKS + lane];
    double r = v.x, i2 = v.y;
    for (int o = 16; o > 0; o >>= 1) {
      r += __shfl_down_sync(0xffffffffu, r, o);
      i2 += __shfl_down_sync(0xffffffffu, i2, o);
    }
    if (lane == 0) g[p] = make_double2(r, i2);
  }
  const int P = a.P, PP = P * P;
  if (tid < P) {
    const double p = P > 1 ? a.norms[3 * tid].x : 1.0;
    const double r = a.eps_pop * exp(-(p / a.eps_pop) * (p / a.eps_pop));
    pop[tid] = p;
    wpm1[tid] = p / (p * p + r * r);
    a.pop[tid] = p;
  }
  // thread (i, j) = (tid % P, tid / P) owns M[i + P j] and its share of multLagDiag
  const int i = tid % P, j = tid / P;
  const bool own = tid < PP;
  if (own) {
    M[tid] = make_double2(0.0, 0.0);
    dterm[tid] = 0.0;
  }
  __syncthreads();
  int base = a.has2 ? PP : 0;
  for (int k = 0; k < a.ndiss1; ++k, base += PP) {
    const cplx* V = g + base;   // V[i + P j] = <A_i|V_k A_j>
    const double ae = a.aeD1[k];
    if (own) {
      const cplx v = V[tid];
      dterm[tid] -= ae * (v.x * v.x + v.y * v.y) * wpm1[i];
      if (i > j) {
        cplx h = make_double2(0.0, 0.0);
        for (int l = 0; l < P; ++l) {
          const cplx t = pk_mul(V[i + P * l], pk_conj(V[j + P * l]));
          h.x += t.x;
          h.y += t.y;
        }
        const double f = ae * (wpm1[i] + wpm1[j]);
        M[tid].x += h.x * f;
        M[tid].y += h.y * f;
      }
      // C[j' + P w] with (j', w) = (i, j): conj(V[w + P j']) scaled by aeD1 WPpopm1_w
      const cplx v2 = pk_conj(V[j + P * i]);
      const double f = ae * wpm1[j];
      a.C1[(long long)k * PP + tid] = make_double2(v2.x * f, v2.y * f);
      a.C2[(long long)k * PP + tid] = make_double2(-v2.y * f, v2.x * f);
    }
  }
  if (a.has2 && own) {
    const cplx* G = g;
    if (i == j) dterm[tid] -= G[tid].x;
    if (i > j) {
      M[tid].x += G[i + P * j].x + G[j + P * i].x;
      M[tid].y += G[i + P * j].y - G[j + P * i].y;
    }
  }
  if (own && i > j) {
    const double dw = pop[i] - pop[j];
    const double r = a.eps_pop * exp(-(dw / a.eps_pop) * (dw / a.eps_pop));
    const double f = dw / (dw * dw + r * r);
    const cplx m = M[tid];
    M[tid] = make_double2(-m.y * f, m.x * f);   // times i f
  }
  __syncthreads();
  if (own) {
    // multLagDiag: the owners' shares added in a fixed order
    double mdiag = 0.0;
    if (i == j)
      for (int q = 0; q < PP; ++q) mdiag += dterm[q];
    // ML = multLagDiag I + i H, H Hermitian from the lower triangle with a zero diagonal
    const cplx h = i > j ? M[tid] : (i < j ? pk_conj(M[j + P * i]) : make_double2(0.0, 0.0));
    a.ML[tid] = make_double2(-h.y + (i == j ? mdiag : 0.0), h.x);
  }
}

void launch_pk_coef(const PkCoefArgs& a, cudaStream_t st) {
  pk_coef_kernel<<<1, 256, sizeof(cplx) * (a.npairs + 1), st>>>(a);
}

__global__ void __launch_bounds__(256) pk_mix_kernel(const PkMix* __restrict__ mix, int nmix,
                                                     const PkState* __restrict__ st, int nstates,
                                                     long long n1tot, int P, cplx* out0) {
  extern __shared__ cplx cm[];   // [nmix][P][P]
  for (int q = threadIdx.x; q < nmix * P * P; q += blockDim.x) cm[q] = mix[q / (P * P)].C[q % (P * P)];
  __syncthreads();
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < n1tot; e += 256LL * gridDim.x) {
    long long c = e;
    int s = 0;
    while (s + 1 < nstates && c >= st[s].n) c -= st[s++].n;
    const long long off = st[s].off + c, n = st[s].n;
    for (int d = 0; d < nmix; ++d) {
      const cplx* in = mix[d].in + off;
      cplx* out = (out0 ? out0 : mix[d].out) + off;
      const cplx* C = cm + d * P * P;
      cplx x[MAX_PACKETS];
      for (int j = 0; j < P; ++j) x[j] = in[j * n];
      for (int w = 0; w < P; ++w) {
        double re = 0.0, im = 0.0;
        for (int j = 0; j < P; ++j) {
          const cplx cc = C[j + P * w];
          re = fma(x[j].x, cc.x, fma(-x[j].y, cc.y, re));
          im = fma(x[j].x, cc.y, fma(x[j].y, cc.x, im));
        }
        if (mix[d].accumulate) {
          const cplx o = out[w * n];
          re += o.x;
          im += o.y;
        }
        out[w * n] = make_double2(re, im);
      }
    }
  }
}

void launch_pk_mix(const PkMix* d_mix, int nmix, const PkState* d_st, int nstates, long long n1tot, int P,
                   cplx* out0, cudaStream_t st) {
  if (nmix <= 0 || n1tot <= 0) return;
  const long long nb = std::min<long long>((n1tot + 255) / 256, FUSED_BLOCKS);
  pk_mix_kernel<<<(int)nb, 256, sizeof(cplx) * nmix * P * P, st>>>(d_mix, nmix, d_st, nstates, n1tot, P, out0);
}
