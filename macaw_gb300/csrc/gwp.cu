// Gaussian (G-MCTDH) block of the equations of motion on the device:
//  - normalised overlaps of multi-dimensional Gaussians (GauOvlMultiD,
//    gmctdh_objects.f90:1497-1519) for S00 and for <Psi1|Psi2>;
//  - one-dimensional integrals <g1|op|g2>/<g1|g2> and <dg1/dxi|op|g2>/<g1|g2>
//    (GauInt1D / Gau10Int1D, hamilton.f90:745-902) and h1mode of a Gaussian
//    mode (hamilton.f90:494-524);
//  - Calc_CY (gmctdh_objects.f90:1198-1333): Sa0, Sa0 S^-1, the matrix C and the
//    vector Y of the parameter equations;
//  - the Tikhonov-regularised solve C x = Y (StdRegSol 'tikh', maths.f90:87-162),
//    dxi = der_factor * x (derivatives.f90:158-173) and the tau matrices of the
//    coefficient correction (derivatives.f90:201-234).
//
// The reference solves C x = Y through the eigen-decomposition of C,
// x = sum_j u_j w_j / (w_j^2 + eps^2) (u_j^H Y).  With w / (w^2 + eps^2) =
// (1 / (w + i eps) + 1 / (w - i eps)) / 2 this is the mean of the solutions of
// (C + i eps) x = Y and (C + i eps)^H x = Y: one LU factorisation with partial
// pivoting, at the condition |C| / eps of C + i eps (the normal equations would square
// it) and without an iterative eigen-solver.  Y is carried as a column and Y^H as a row
// of the factorisation, so only the two back-substitutions remain.
#include <float.h>

#include <algorithm>

#include "kernels.cuh"
#include "fixed.cuh"

namespace {

__device__ __forceinline__ cplx cexp_(cplx z) {
  const double e = exp(z.x);
  double s, c;
  sincos(z.y, &s, &c);
  return mkc(e * c, e * s);
}
__device__ __forceinline__ cplx neg_i(cplx z) { return mkc(z.y, -z.x); }   // -i z
__device__ __forceinline__ cplx cdivr(cplx z, double r) { return mkc(z.x / r, z.y / r); }
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  const double d = b.x * b.x + b.y * b.y;
  return mkc((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}

// T(k, n) = binomial(n, 2k) * (2k-1)!!, the moment coefficients of hamilton.f90:761-785
// (every intermediate of the product formula is an exact integer below 2^53).
__device__ double gau_coeff(int k, int n) {
  double b = 1.0;
  for (int i = 0; i < 2 * k; ++i) b = b * (double)(n - i) / (double)(i + 1);
  double df = 1.0;
  for (int x = 2 * k - 1; x > 0; x -= 2) df *= (double)x;
  return b * df;
}
__device__ cplx cpow_int(cplx z, int m) {
  cplx r = mkc(1.0, 0.0);
  for (int i = 0; i < m; ++i) r = cmul(r, z);
  return r;
}
__device__ double rpow_int(double z, int m) {
  double r = 1.0;
  for (int i = 0; i < m; ++i) r *= z;
  return r;
}

// <g1|op|g2>/<g1|g2> for g = exp(a x^2 + xi x) and the primitive operator code iop
// (0 identity, -1 p, -2 d^2/dq^2, -3 qp, k >= 1: q^k).
__device__ cplx gau_int_1d(double a1, double a2, cplx xi1, cplx xi2, int iop) {
  const cplx x1c = cconj(xi1);
  const double a12 = a1 + a2;
  switch (iop) {
    case 0:
      return mkc(1.0, 0.0);
    case -1: {
      const cplx num = csub(cscale(xi2, a1), cscale(x1c, a2));
      return cdivr(neg_i(num), a12);
    }
    case -2: {
      const cplx u = cdivr(csub(cscale(x1c, a2), cscale(xi2, a1)), a12);
      return cadd(cmul(u, u), mkc(2.0 * a1 * a2 / a12, 0.0));
    }
    case -3: {
      const cplx g = cadd(mkc(a1 * a1 - a2 * a2, 0.0), cmul(csub(cscale(x1c, a2), cscale(xi2, a1)), cadd(x1c, xi2)));
      return cdivr(neg_i(g), a12 * a12);
    }
    case 1:
      return cdivr(cadd(x1c, xi2), -2.0 * a12);
    case 2: {
      const double a = 2.0 * a12;
      const cplx v = cdivr(cadd(x1c, xi2), a);
      return csub(cmul(v, v), mkc(1.0 / a, 0.0));
    }
    default:
      break;
  }
  const cplx c1 = cadd(x1c, xi2);
  const double an = -2.0 * a12;
  if (iop >= 3 && iop <= 19 && (iop & 1)) {
    cplx g = mkc(0.0, 0.0);
    for (int k = 0; k <= iop / 2; ++k) {
      const double f = gau_coeff(k, iop) / rpow_int(an, iop - k);
      g = cadd(g, cscale(cpow_int(c1, iop - 2 * k), f));
    }
    return g;
  }
  if (iop >= 4 && iop <= 20 && !(iop & 1)) {
    const cplx c2 = cdivr(cmul(c1, c1), an);
    cplx p = mkc(1.0, 0.0);
    cplx g = mkc(0.0, 0.0);
    for (int k = iop / 2; k >= 0; --k) {
      g = cadd(g, cscale(p, gau_coeff(k, iop)));
      p = cmul(p, c2);
    }
    return cdivr(g, rpow_int(an, iop / 2));
  }
  return mkc(nan(""), 0.0);   // unsupported codes are rejected when the plan is built
}

// <dg1/dxi1|op|g2>/<g1|g2> (Gau10Int1D)
__device__ cplx gau10_int_1d(double a1, double a2, cplx xi1, cplx xi2, int iop) {
  if (iop == -1) {
    const cplx t1 = neg_i(cmul(xi2, gau_int_1d(a1, a2, xi1, xi2, 1)));
    const cplx t2 = cscale(neg_i(gau_int_1d(a1, a2, xi1, xi2, 2)), 2.0 * a2);
    return cadd(t1, t2);
  }
  if (iop == -2) {
    const cplx g1 = gau_int_1d(a1, a2, xi1, xi2, 1);
    const cplx g2 = gau_int_1d(a1, a2, xi1, xi2, 2);
    const cplx g3 = gau_int_1d(a1, a2, xi1, xi2, 3);
    cplx r = cmul(cadd(mkc(a2 + a2, 0.0), cmul(xi2, xi2)), g1);
    r = cadd(r, cmul(cscale(xi2, 4.0 * a2), g2));
    return cadd(r, cscale(g3, 4.0 * a2 * a2));
  }
  if (iop == -3) {
    const cplx g1 = gau_int_1d(a1, a2, xi1, xi2, 1);
    const cplx g2 = gau_int_1d(a1, a2, xi1, xi2, 2);
    const cplx g3 = gau_int_1d(a1, a2, xi1, xi2, 3);
    return neg_i(cadd(cadd(g1, cmul(cscale(xi2, 2.0), g2)), cscale(g3, 4.0 * a2)));
  }
  return gau_int_1d(a1, a2, xi1, xi2, iop + 1);
}

// Normalised overlap of two nmd-dimensional Gaussians.
__device__ cplx gau_ovl(const double* a1, const double* a2, const cplx* xi1, const cplx* xi2, int nmd) {
  bool same = true;
  for (int k = 0; k < nmd; ++k)
    if (!(fabs(a1[k] - a2[k]) < DBL_EPSILON)) same = false;
  cplx c = mkc(0.0, 0.0);
  if (same) {
    for (int k = 0; k < nmd; ++k) {
      const cplx s = cadd(cconj(xi1[k]), xi2[k]);
      const cplx t = csub(mkc(xi1[k].x * xi1[k].x + xi2[k].x * xi2[k].x, 0.0), cscale(cmul(s, s), 0.5));
      c = cadd(c, cdivr(t, a1[k]));
    }
    return cexp_(cscale(c, 0.25));
  }
  double d = 1.0;
  for (int k = 0; k < nmd; ++k) {
    const cplx s = cadd(cconj(xi1[k]), xi2[k]);
    const double a12 = a1[k] + a2[k];
    c = cadd(c, mkc(xi1[k].x * xi1[k].x / a1[k] + xi2[k].x * xi2[k].x / a2[k], 0.0));
    c = csub(c, cdivr(cmul(s, s), a12));
    d *= 4.0 * a1[k] * a2[k] / (a12 * a12);
  }
  return cscale(cexp_(cscale(c, 0.25)), sqrt(sqrt(d)));
}

// A warp per 32 entries: an entry is a serial chain of FP64 divisions (443 cycles each)
// and exponentials, so the warps go to as many sub-partitions as there are (four
// 32 x 32 overlaps of 12 DOFs: 509 us with a block of eight warps each, 76 now).
__global__ void __launch_bounds__(32) gwp_ovl_kernel(const GwpOvlDesc* __restrict__ descs) {
  const GwpOvlDesc& d = descs[blockIdx.x];
  for (int e = blockIdx.y * 32 + threadIdx.x; e < d.n1 * d.n2; e += 32 * gridDim.y) {
    const int j1 = e % d.n1, j2 = e / d.n1;
    cplx v;
    if (d.kind == 3) {
      // Calc_Err_SPF (cmf2_derivatives.f90:301-315): 2 - 2 Re<g(x)|g(y)> on the
      // diagonal, S(x,x) + S(y,y) - S(x,y) - S(y,x) above it
      if (j1 > j2) continue;
      const double* a1 = d.a + d.lda * j1;
      const double* a2 = d.a + d.lda * j2;
      const cplx* x1 = d.xi1 + d.nmd * j1;
      const cplx* x2 = d.xi1 + d.nmd * j2;
      const cplx* y1 = d.xi2 + d.nmd * j1;
      const cplx* y2 = d.xi2 + d.nmd * j2;
      if (j1 == j2) {
        v = mkc(2.0 - 2.0 * gau_ovl(a1, a1, x1, y1, d.nmd).x, 0.0);
      } else {
        v = cadd(gau_ovl(a1, a2, x1, x2, d.nmd), gau_ovl(a1, a2, y1, y2, d.nmd));
        v = csub(v, gau_ovl(a1, a2, x1, y2, d.nmd));
        v = csub(v, gau_ovl(a1, a2, y1, x2, d.nmd));
      }
    } else if (d.kind == 0 && j1 == j2) {
      v = mkc(1.0, 0.0);
    } else if (d.kind == 0 && j1 > j2) {
      v = cconj(gau_ovl(d.a + d.lda * j2, d.a + d.lda * j1, d.xi1 + d.nmd * j2, d.xi2 + d.nmd * j1, d.nmd));
    } else if (d.kind == 2) {
      v = cconj(gau_ovl(d.a + d.lda * j2, d.a + d.lda * j1, d.xi2 + d.nmd * j2, d.xi1 + d.nmd * j1, d.nmd));
    } else {
      v = gau_ovl(d.a + d.lda * j1, d.a + d.lda * j2, d.xi1 + d.nmd * j1, d.xi2 + d.nmd * j2, d.nmd);
    }
    d.out[e] = v;
  }
}

__device__ cplx gwp_h1_entry(const GwpH1Desc& d, int j1, int j2) {
  cplx g = mkc(1.0, 0.0);
  for (int k = 0; k < d.nmd; ++k)
    g = cmul(g, gau_int_1d(d.a[k + d.lda * j1], d.a[k + d.lda * j2], d.xi1[k + d.nmd * j1], d.xi2[k + d.nmd * j2],
                           d.ops[k]));
  return cmul(d.S[j1 + d.n1 * j2], g);
}

__global__ void __launch_bounds__(64) gwp_h1_kernel(const GwpH1Desc* __restrict__ descs) {
  const GwpH1Desc& d = descs[blockIdx.x];
  for (int e = blockIdx.y * 64 + threadIdx.x; e < d.n1 * d.n2; e += 64 * gridDim.y) {
    const int j1 = e % d.n1, j2 = e / d.n1;
    d.out[e] = (d.same_state && j1 > j2) ? cconj(gwp_h1_entry(d, j2, j1)) : gwp_h1_entry(d, j1, j2);
  }
}

// Sa0 (nG x n): <dg_j1/dxi_k | g_j2> / normalisation, upper blocks from the
// integrals and the lower ones as conjugates (gmctdh_objects.f90:1218-1240).
__global__ void gwp_sa0_kernel(const GwpCYDesc* __restrict__ descs) {
  const GwpCYDesc& d = descs[blockIdx.y];
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.nG * d.n) return;
  const int r = e % d.nG, j2 = e / d.nG;
  const int j1 = r / d.nmd, k = r % d.nmd;
  cplx v;
  if (j1 <= j2) {
    v = cmul(d.S[j1 + d.n * j2], gau_int_1d(d.a[k + d.lda * j1], d.a[k + d.lda * j2], d.xi[k + d.nmd * j1],
                                            d.xi[k + d.nmd * j2], 1));
  } else {
    v = cconj(cmul(d.S[j2 + d.n * j1], gau_int_1d(d.a[k + d.lda * j2], d.a[k + d.lda * j1], d.xi[k + d.nmd * j2],
                                                  d.xi[k + d.nmd * j1], 1)));
  }
  d.Sa0[e] = v;
}

// Sa0Sm1 = Sa0 * S^-1 (nG x n)
__global__ void gwp_sa0sm1_kernel(const GwpCYDesc* __restrict__ descs) {
  const GwpCYDesc& d = descs[blockIdx.y];
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.nG * d.n) return;
  const int r = e % d.nG, j = e / d.nG;
  cplx s = mkc(0.0, 0.0);
  for (int l = 0; l < d.n; ++l) cfma(s, d.Sa0[r + d.nG * l], d.Sm1[l + d.n * j]);
  d.Sa0Sm1[e] = s;
}

// Upper-triangle entry (r <= c) of C = rho o (Sab - (Sa0Sm1 Sa0^H + Sa0 Sa0Sm1^H)/2)
// (gmctdh_objects.f90:1242-1283).
__device__ cplx gwp_c_entry(const GwpCYDesc& d, int r, int c) {
  const int j1 = r / d.nmd, k1 = r % d.nmd, j2 = c / d.nmd, k2 = c % d.nmd;
  const double* a = d.a;
  const cplx* xi = d.xi;
  cplx v;
  if (k1 == k2) {
    v = gau_int_1d(a[k1 + d.lda * j1], a[k2 + d.lda * j2], xi[k1 + d.nmd * j1], xi[k2 + d.nmd * j2], 2);
  } else {
    const cplx g1 = gau_int_1d(a[k1 + d.lda * j1], a[k1 + d.lda * j2], xi[k1 + d.nmd * j1], xi[k1 + d.nmd * j2], 1);
    const cplx g2 = gau_int_1d(a[k2 + d.lda * j1], a[k2 + d.lda * j2], xi[k2 + d.nmd * j1], xi[k2 + d.nmd * j2], 1);
    v = cmul(g1, g2);
  }
  cplx sab = cmul(d.S[j1 + d.n * j2], v);
  cplx s1 = mkc(0.0, 0.0), s2 = mkc(0.0, 0.0);
  for (int j = 0; j < d.n; ++j) {
    cfma(s1, d.Sa0Sm1[r + d.nG * j], cconj(d.Sa0[c + d.nG * j]));
    cfma(s2, d.Sa0[r + d.nG * j], cconj(d.Sa0Sm1[c + d.nG * j]));
  }
  sab = csub(sab, cscale(cadd(s1, s2), 0.5));
  return cmul(d.rho[j1 + d.n * j2], sab);
}

// C + i eps into the bordered system [C + i eps, Y; Y^H, 0], the Hermitian C from its
// upper triangle (an element costs about 320 FP64 instructions: 64 n for the projection).
__global__ void __launch_bounds__(64) gwp_c_kernel(const GwpCYDesc* __restrict__ descs) {
  const GwpCYDesc& d = descs[blockIdx.z];
  const int r0 = 8 * blockIdx.x, c0 = 8 * blockIdx.y;
  if (r0 > c0) return;
  const int r = r0 + (threadIdx.x & 7), c = c0 + (threadIdx.x >> 3);
  if (r > c || c >= d.nG) return;
  const long long ld = d.nG + 1LL;
  cplx v = gwp_c_entry(d, r, c);
  if (r == c)
    v.y += d.eps;
  else
    d.M[c + ld * r] = cconj(v);
  d.M[r + ld * c] = v;
}

// Y (gmctdh_objects.f90:1285-1326): per entry r = j1*nmd + k, the sum over operators and
// j2 of MF(j1,j2) (Ha0 - Sa0Sm1 h)(r, j2).  The second part is summed over the operators
// first, G(j, j1) = sum MF(j1, j2) h(j, j2), and multiplied by Sa0Sm1 once: n^2 products
// per operator instead of n^2 nmd.
// Stage 1a: a thread per (j1, j2, YOP_CHUNK operators) computes the pair's <q_k> once, the
// integrals of each operator's acting DOFs, and the nmd sums over its operators into
// part[(chunk*maxn2 + j2)*nG + r].
// Stage 1b: a thread per (j, j1, operator) sums its part of G over j2.
// Stage 2: a warp per r adds the terms in a fixed order.
#define YOP_CHUNK 4
__global__ void __launch_bounds__(32) gwp_y_part_kernel(const GwpCYDesc* __restrict__ descs,
                                                        const GwpYOp* __restrict__ ops, cplx* __restrict__ part,
                                                        long long part_ld, int maxn2) {
  const GwpCYDesc& d = descs[blockIdx.y];
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nch = (d.op_count + YOP_CHUNK - 1) / YOP_CHUNK;
  if (e >= (long long)d.n * maxn2 * nch) return;
  const int j1 = (int)(e % d.n);
  const int j2 = (int)((e / d.n) % maxn2);
  const int ch = (int)(e / ((long long)d.n * maxn2));
  const int nmd = d.nmd;
  const double* a = d.a;
  cplx q1[GWP_MAXDOF], acc[GWP_MAXDOF];
  const cplx* xi2 = nullptr;   // q1 is of this right state
#pragma unroll
  for (int k = 0; k < GWP_MAXDOF; ++k) acc[k] = mkc(0.0, 0.0);
  for (int o = ch * YOP_CHUNK; o < min(d.op_count, (ch + 1) * YOP_CHUNK); ++o) {
    const GwpYOp& op = ops[d.op_first + o];
    if (j2 >= op.n2) continue;
    if (op.xi2 != xi2) {
      xi2 = op.xi2;
#pragma unroll
      for (int k = 0; k < GWP_MAXDOF; ++k)
        if (k < nmd)
          q1[k] = gau_int_1d(a[k + d.lda * j1], a[k + d.lda * j2], d.xi[k + d.nmd * j1], xi2[k + d.nmd * j2], 1);
    }
    const cplx w0 = cmul(op.mf[j1 + d.n * j2], op.S12[j1 + d.n * j2]);
    // DOFs without an operator: the product of all acting integrals times <q_k>
    cplx w = w0;
    for (int k = 0; k < nmd; ++k)
      if (op.ops[k] != 0)
        w = cmul(w, gau_int_1d(a[k + d.lda * j1], a[k + d.lda * j2], d.xi[k + d.nmd * j1], xi2[k + d.nmd * j2], op.ops[k]));
#pragma unroll
    for (int k = 0; k < GWP_MAXDOF; ++k) {
      if (k >= nmd) break;
      if (op.ops[k] == 0) {
        cfma(acc[k], w, q1[k]);
      } else {
        cplx v = cmul(w0, gau10_int_1d(a[k + d.lda * j1], a[k + d.lda * j2], d.xi[k + d.nmd * j1], xi2[k + d.nmd * j2],
                                       op.ops[k]));
        for (int q = 0; q < nmd; ++q)
          if (q != k && op.ops[q] != 0)
            v = cmul(v, gau_int_1d(a[q + d.lda * j1], a[q + d.lda * j2], d.xi[q + d.nmd * j1], xi2[q + d.nmd * j2],
                                   op.ops[q]));
        acc[k] = cadd(acc[k], v);
      }
    }
  }
  cplx* out = part + (long long)blockIdx.y * part_ld + ((long long)ch * maxn2 + j2) * d.nG + (long long)j1 * nmd;
#pragma unroll
  for (int k = 0; k < GWP_MAXDOF; ++k)
    if (k < nmd) out[k] = acc[k];
}

// part of G behind the terms of stage 1a: [operator][j1][j]
__global__ void __launch_bounds__(32) gwp_y_mf_kernel(const GwpCYDesc* __restrict__ descs,
                                                      const GwpYOp* __restrict__ ops, cplx* __restrict__ part,
                                                      long long part_ld, long long g_off) {
  const GwpCYDesc& d = descs[blockIdx.z];
  const int o = blockIdx.y;
  if (o >= d.op_count) return;
  const int e = blockIdx.x * 32 + threadIdx.x, j = e % d.n, j1 = e / d.n;
  if (j1 >= d.n) return;
  const GwpYOp& op = ops[d.op_first + o];
  cplx v = mkc(0.0, 0.0);
  for (int j2 = 0; j2 < op.n2; ++j2) cfma(v, op.mf[j1 + d.n * j2], op.h[j + d.n * j2]);
  part[(long long)blockIdx.z * part_ld + g_off + ((long long)o * d.n + j1) * d.n + j] = v;
}

__device__ cplx warp_sum(cplx v);

__global__ void __launch_bounds__(32) gwp_y_sum_kernel(const GwpCYDesc* __restrict__ descs,
                                                       const cplx* __restrict__ part, long long part_ld,
                                                       long long g_off, int maxn2) {
  const GwpCYDesc& d = descs[blockIdx.y];
  const int r = blockIdx.x, lane = threadIdx.x;
  if (r >= d.nG) return;
  const cplx* base = part + (long long)blockIdx.y * part_ld;
  const int j1 = r / d.nmd, nterm = (d.op_count + YOP_CHUNK - 1) / YOP_CHUNK * maxn2;
  cplx acc = mkc(0.0, 0.0);
#pragma unroll 4
  for (int t = lane; t < nterm; t += 32) acc = cadd(acc, base[(long long)t * d.nG + r]);
  if (lane < d.n) {   // n <= 32
    const cplx* g = base + g_off + (long long)j1 * d.n + lane;
    cplx s = mkc(0.0, 0.0);
#pragma unroll 4
    for (int o = 0; o < d.op_count; ++o) s = cadd(s, g[(long long)o * d.n * d.n]);
    acc = csub(acc, cmul(d.Sa0Sm1[r + d.nG * lane], s));
  }
  acc = warp_sum(acc);
  if (lane) return;
  const long long ld = d.nG + 1LL;
  d.M[r + ld * d.nG] = acc;
  d.M[d.nG + ld * r] = cconj(acc);
  if (r == 0) d.M[d.nG + ld * d.nG] = mkc(0.0, 0.0);
}

__device__ cplx warp_sum(cplx v) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  v.x = __shfl_sync(0xffffffffu, v.x, 0);
  v.y = __shfl_sync(0xffffffffu, v.y, 0);
  return v;
}

// LU factorisation of the bordered system in panels of LU_PW columns, two launches per
// panel (384 unknowns, two systems: 48 panels of 17.5 and updates of 9.0 us,
// where a Householder QR of [C; eps I] took 48 launches of 127).
//
// Panel: one block per system, a row of the panel per thread in registers.  Rows stay
// where they are; perm lists them in pivot order, act the rows not yet taken (the last
// is the border row, never a pivot).  M keeps the multipliers, R receives U in pivot
// order.  Bound by the serial pivots and one SM's FP64 pipe (4 + 4 (PW - k) FMAs per row).
__global__ void __launch_bounds__(LU_MAXROWS) lu_panel_kernel(const GwpCYDesc* __restrict__ descs, int j0) {
  const GwpCYDesc& d = descs[blockIdx.x];
  const int nG = d.nG;
  if (j0 >= nG) return;
  const int pw = min(LU_PW, nG - j0);
  const long long ld = nG + 1;
  const int r = threadIdx.x, lane = r & 31, warp = r >> 5, nw = blockDim.x >> 5;
  __shared__ cplx prow[LU_PW + 1];       // the pivot row and the pivot's reciprocal
  __shared__ unsigned wmax[32];
  __shared__ int wrow[32];
  bool act = r <= nG && (j0 == 0 || d.step[r] < 0);
  const bool start = act;
  int step = -1;
  cplx a[LU_PW];
#pragma unroll
  for (int j = 0; j < LU_PW; ++j) a[j] = act && j < pw ? d.M[r + ld * (j0 + j)] : mkc(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < LU_PW; ++k) {
    if (k >= pw) break;
    // the largest remaining element of the column (by its larger component's leading word)
    const unsigned mag = act && r < nG ? fx_mag(a[k]) + 1u : 0u;
    const unsigned m = __reduce_max_sync(0xffffffffu, mag);
    const unsigned who = __ballot_sync(0xffffffffu, mag == m);
    if (lane == 0) {
      wmax[warp] = m;
      wrow[warp] = 32 * warp + __ffs(who) - 1;
    }
    __syncthreads();
    const unsigned v = lane < nw ? wmax[lane] : 0u;
    const int win = wrow[__ffs(__ballot_sync(0xffffffffu, v == __reduce_max_sync(0xffffffffu, v))) - 1];
    if (r == win) {
      act = false;
      step = j0 + k;
      const double q = 1.0 / fma(a[k].x, a[k].x, a[k].y * a[k].y);
      prow[LU_PW] = mkc(a[k].x * q, -a[k].y * q);
#pragma unroll
      for (int j = k + 1; j < LU_PW; ++j) prow[j] = a[j];
    }
    __syncthreads();
    if (act) {
      const cplx w = cmul(a[k], prow[LU_PW]);
      a[k] = w;
#pragma unroll
      for (int j = k + 1; j < LU_PW; ++j) {
        const cplx u = prow[j];
        a[j].x = fma(-w.x, u.x, fma(w.y, u.y, a[j].x));
        a[j].y = fma(-w.x, u.y, fma(-w.y, u.x, a[j].y));
      }
    }
    if (r == win) d.rdiag[j0 + k] = prow[LU_PW];
  }
  if (start) {
    d.step[r] = step;
    if (step >= 0) d.perm[step] = r;
#pragma unroll
    for (int j = 0; j < LU_PW; ++j) {
      if (j >= pw) break;
      d.M[r + ld * (j0 + j)] = a[j];
      if (step >= 0 && j0 + j >= step) d.R[step + (long long)nG * (j0 + j)] = a[j];
    }
  }
  const unsigned bal = __ballot_sync(0xffffffffu, act);
  __syncthreads();
  if (lane == 0) wrow[warp] = __popc(bal);
  __syncthreads();
  if (act) {
    int pos = __popc(bal & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) pos += wrow[w];
    d.act[pos] = r;
  }
}

// Trailing update: a block takes 32 of the remaining rows and 32 of the remaining
// columns (the right-hand side is the last).  It solves the panel's unit lower triangle
// for its columns (the blocks of the first row of blocks store the result as U), then
// subtracts the rank-8 product as digit products (fixed.cuh; a warp's 16 rows are
// the MMA's rows, the (re, im) of four columns its columns, as in the mode products),
// where FP64 would take 18 us of an SM's FP64 pipe per block; elements small against the
// factors (a panel whose rows and columns are graded) are done in FP64.
__global__ void __launch_bounds__(256) lu_update_kernel(const GwpCYDesc* __restrict__ descs, int j0) {
  constexpr int NS = FX_NS, SH = fx_headroom(LU_PW);
  const GwpCYDesc& d = descs[blockIdx.z];
  const int nG = d.nG;
  if (j0 >= nG) return;
  const int pw = min(LU_PW, nG - j0);
  const long long ld = nG + 1;
  const int mrows = nG - j0 - pw + 1, c0 = j0 + pw;
  const int i0 = 32 * blockIdx.y;
  if (i0 >= mrows || c0 + 32 * (int)blockIdx.x > nG) return;
  __shared__ cplx Ls[LU_PW][LU_PW];
  __shared__ cplx T[32][LU_PW + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  int row[2];
  cplx x[2][2];
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int i = i0 + 16 * (warp & 1) + g + 8 * f;
    row[f] = i < mrows ? d.act[i] : -1;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      x[f][k] = row[f] >= 0 && 4 * k + q < pw ? d.M[row[f] + ld * (j0 + 4 * k + q)] : mkc(0.0, 0.0);
  }
  {
    const int i = tid & 7, cc = tid >> 3, col = c0 + 32 * blockIdx.x + cc;
    const int row = i < pw ? d.perm[j0 + i] : 0;
    cplx t = i < pw && col <= nG ? d.M[row + ld * col] : mkc(0.0, 0.0);
    if (cc < LU_PW) Ls[i][cc] = cc < i && i < pw ? d.M[row + ld * (j0 + cc)] : mkc(0.0, 0.0);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LU_PW - 1; ++k) {
      const cplx u = mkc(__shfl_sync(0xffffffffu, t.x, (lane & 24) + k), __shfl_sync(0xffffffffu, t.y, (lane & 24) + k));
      const cplx w = Ls[i][k];
      if (i > k) {
        t.x = fma(-w.x, u.x, fma(w.y, u.y, t.x));
        t.y = fma(-w.x, u.y, fma(-w.y, u.x, t.y));
      }
    }
    T[cc][i] = t;
    if (i0 == 0 && i < pw && col <= nG) d.R[j0 + i + (long long)nG * col] = t;
  }
  __syncthreads();
  unsigned er[2];
  bool bad = false, live[2];
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    unsigned mag = max(fx_mag(x[f][0]), fx_mag(x[f][1]));
    mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 1));
    mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 2));
    bad = bad || !fx_ok(mag);
    live[f] = mag != 0u;
    er[f] = fx_ebits(mag);
  }
  cplx y[2][2];   // in flight during the products
#pragma unroll
  for (int tt = 0; tt < 2; ++tt)
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const int col = c0 + 32 * blockIdx.x + 4 * (2 * (warp >> 1) + tt) + q;
      y[tt][f] = row[f] >= 0 && col <= nG ? d.M[row[f] + ld * col] : mkc(0.0, 0.0);
    }
  unsigned A[NS][4];
#pragma unroll
  for (int f = 0; f < 2; ++f)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      unsigned s[NS];
      fx_digits(x[f][k].x, x[f][k].y, er[f], er[f], s);
#pragma unroll
      for (int i = 0; i < NS; ++i) A[i][2 * k + f] = s[i];
    }
#pragma unroll
  for (int tt = 0; tt < 2; ++tt) {
    const int t = 2 * (warp >> 1) + tt, jo = 4 * t + (g >> 1);
    const cplx m0 = T[jo][q], m1 = T[jo][4 + q];
    unsigned mag = max(fx_mag(m0), fx_mag(m1));
    mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 1));
    mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, 2));
    const bool slow = __any_sync(0xffffffffu, bad || !fx_ok(mag));
    const unsigned ec = fx_ebits(mag);
    const unsigned ecol = __shfl_sync(0xffffffffu, ec, 8 * q), es = fx_exp(ecol, 0u, 44 + SH);
    const bool lcol = __shfl_sync(0xffffffffu, mag, 8 * q) != 0u;
    const int col = c0 + 32 * blockIdx.x + 4 * t + q;
    float c[NS][4];
    if (!slow) {
      unsigned s0[NS], s1[NS];
      fx_digits(m0.x, m0.y, ec, ec, s0);
      fx_digits(m1.x, m1.y, ec, ec, s1);
#pragma unroll
      for (int i = 0; i < NS; ++i) {   // column re: (Mr, -Mi); column im: (Mi, Mr)
        const unsigned w0 = (g & 1) ? __byte_perm(s0[i], s0[i], 0x1032) : s0[i] ^ 0x80000000u;
        const unsigned w1 = (g & 1) ? __byte_perm(s1[i], s1[i], 0x1032) : s1[i] ^ 0x80000000u;
#pragma unroll
        for (int j = 0; j + i < NS; ++j) fx_mma16(c[i + j], A[j], w0, w1, i == 0);
      }
    }
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (row[f] < 0 || col > nG) continue;
      cplx v = mkc(0.0, 0.0);
      bool fp64 = slow;
      if (!slow) {
        const long long re = fx_join(c, 2 * f, fx_pow2(SH)), im = fx_join(c, 2 * f + 1, fx_pow2(SH));
        v = mkc(fx_double(re, es + er[f]), fx_double(im, es + er[f]));
        // both the product and the element below 2^-8 of the largest factors' product
        fp64 = fx_small(re, im, fx_small_limit(SH)) && live[f] && lcol && fx_mag(y[tt][f]) < er[f] + ecol - (1029u << 20);
      }
      if (fp64) {
        v = mkc(0.0, 0.0);
        for (int k = 0; k < pw; ++k) cfma(v, d.M[row[f] + ld * (j0 + k)], T[4 * t + q][k]);
      }
      d.M[row[f] + ld * col] = csub(y[tt][f], v);
    }
  }
}

// Back-substitutions U x = L^-1 P Y (system 0) and L^H P x = U^-H Y (system 1), a block
// each: blocks of eight unknowns from the last, warp 0 solving the next block while the
// other warps update the rest (one barrier per eight unknowns; the former column-wise
// form, with a division and two barriers per unknown, took 878 us at 384 unknowns).
__global__ void __launch_bounds__(512) lu_back_kernel(const GwpCYDesc* __restrict__ descs) {
  extern __shared__ cplx z[];
  const GwpCYDesc& d = descs[blockIdx.y];
  const int nG = d.nG, sys = blockIdx.x;
  const long long ld = nG + 1;
  int* prm = reinterpret_cast<int*>(z + nG);
  const int tid = threadIdx.x, lane = tid & 31;
  for (int k = tid; k < nG; k += blockDim.x) {
    prm[k] = d.perm[k];
    z[k] = sys == 0 ? d.R[k + (long long)nG * nG] : cconj(d.M[nG + ld * k]);
  }
  __syncthreads();
  // coefficient of unknown k in the equation of unknown i < k
  auto coef = [&](int i, int k) {
    return sys == 0 ? d.R[i + (long long)nG * k] : cconj(d.M[prm[k] + ld * i]);
  };
  auto less = [&](cplx& v, cplx c, cplx x) {
    v.x = fma(-c.x, x.x, fma(c.y, x.y, v.x));
    v.y = fma(-c.x, x.y, fma(-c.y, x.x, v.y));
  };
  const int nb = (nG + 7) >> 3;
  for (int b = nb; b >= 1; --b) {
    // unknowns 8 b .. are known; warp 0: the block's share of them, then the block before
    const int k0 = 8 * b, kn = min(8, nG - k0);
    if (tid < 32) {
      const int i0 = k0 - 8, i = i0 + (lane & 7), kq = lane >> 3;
      const bool on = i < nG;
      // lane (i, kq): unknowns kq, kq + 4 of either block
      cplx cd[2], cu[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = kq + 4 * h;
        cd[h] = on && i0 + k < nG && i0 + k > i ? coef(i, i0 + k) : mkc(0.0, 0.0);
        cu[h] = on && k < kn ? coef(i, k0 + k) : mkc(0.0, 0.0);
      }
      cplx v = kq == 0 && on ? z[i] : mkc(0.0, 0.0);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (kq + 4 * h < kn) less(v, cu[h], z[k0 + kq + 4 * h]);
#pragma unroll
      for (int o = 8; o < 32; o <<= 1)
        v = cadd(v, mkc(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)));
      if (sys == 0) {   // rows divided by the diagonal ahead of the chain
        const cplx rd = on ? d.rdiag[i] : mkc(0.0, 0.0);
        v = cmul(v, rd);
        cd[0] = cmul(cd[0], rd);
        cd[1] = cmul(cd[1], rd);
      }
#pragma unroll
      for (int k = 7; k > 0; --k) {
        const int src = (lane & 7) + 8 * (k & 3);
        const cplx c = mkc(__shfl_sync(0xffffffffu, cd[k >> 2].x, src), __shfl_sync(0xffffffffu, cd[k >> 2].y, src));
        const cplx x = mkc(__shfl_sync(0xffffffffu, v.x, k), __shfl_sync(0xffffffffu, v.y, k));
        less(v, c, x);   // c = 0 for unknowns k ..
      }
      if (kq == 0 && on) z[i] = v;
    } else if ((tid >> 5) & 3) {   // the sub-partition of warp 0 is left to it
      for (int r = 96 * (tid >> 7) + ((tid >> 5 & 3) - 1) * 32 + lane; r < k0 - 8; r += 96 * (blockDim.x >> 7)) {
        cplx v = z[r], cf[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) cf[k] = k < kn ? coef(r, k0 + k) : mkc(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < kn) less(v, cf[k], z[k0 + k]);
        z[r] = v;
      }
    }
    __syncthreads();
  }
  for (int k = tid; k < nG; k += blockDim.x) d.x[sys == 0 ? k : nG + prm[k]] = z[k];
}

// x = the mean of the two solutions, dxi = der * x, and tau
// tau(j1, j2) = sum_k conj(Sa0Sm1(j2*nmd+k, j1)) dxi(k, j2) + diagonal phase term
__global__ void __launch_bounds__(256) gwp_tau_kernel(const GwpCYDesc* __restrict__ descs, cplx der,
                                                      cplx* __restrict__ out, int* status) {
  extern __shared__ cplx dx[];
  const GwpCYDesc& d = descs[blockIdx.y];
  const int nG = d.nG;
  for (int r = threadIdx.x; r < nG; r += blockDim.x) {
    cplx x = cscale(cadd(d.x[r], d.x[nG + r]), 0.5);
    if (!isfinite(x.x) || !isfinite(x.y)) {
      if (blockIdx.x == 0) atomicOr(status, DEVST_NONFINITE);
      x = mkc(0.0, 0.0);
    }
    dx[r] = cmul(der, x);
    if (blockIdx.x == 0) out[d.dxi_offset + r] = dx[r];
  }
  __syncthreads();
  const int n = d.n, nmd = d.nmd;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += gridDim.x * blockDim.x) {
    const int j1 = e % n, j2 = e / n;
    cplx t = mkc(0.0, 0.0);
    for (int k = 0; k < nmd; ++k) cfma_conj(t, d.Sa0Sm1[(j2 * nmd + k) + (long long)nG * j1], dx[k + nmd * j2]);
    if (j1 == j2) {
      double dd = 0.0;
      for (int k = 0; k < nmd; ++k) dd += d.xi[k + nmd * j2].x * dx[k + nmd * j2].x / d.a[k + d.lda * j2];
      t.x += dd * 0.5;
    }
    d.tau[e] = t;
  }
}

// Tikhonov-regularised inverse of a Hermitian n x n matrix (n <= 32), X = (A^2 + eps^2)^-1 A,
// the matrix StdRegInv 'tikh' (maths.f90:8-83) builds from the eigen-decomposition
// U w/(w^2 + eps^2) U^H: the Hermitian part of (A + i eps)^-1.  Gauss-Jordan exchanges
// with partial pivoting, an element per thread (a warp holds a column, a lane a row),
// one barrier per pivot: the warp of the next column updates it, finds the pivot and
// publishes the multipliers while the others still update.  Bound by the FP64 pipe (four
// instructions per element and pivot) and the serial pivots; two 32 x 32 inverses took
// 710 us as a Householder QR of [A; eps I], 57 now.
__global__ void __launch_bounds__(1024) tikh_inv_kernel(const RegInvDesc* __restrict__ descs) {
  __shared__ cplx mult[2][MAXN_SPF];      // multipliers; the pivot row's is minus the reciprocal
  __shared__ int s_row[MAXN_SPF];         // pivot row of each step
  __shared__ cplx X[MAXN_SPF][MAXN_SPF + 1];
  const RegInvDesc& d = descs[blockIdx.x];
  const int n = d.n, i = threadIdx.x & 31, j = threadIdx.x >> 5;   // a column per warp; blockDim.x = 32 max n
  cplx a = mkc(0.0, 0.0);
  if (i < n && j < n) {
    // the upper triangle is authoritative (zheev 'U'): mirror it, real diagonal
    a = (i <= j) ? d.A[i + n * j] : cconj(d.A[j + n * i]);
    if (i == j) a.y = d.eps;
  }
  bool taken = i >= n;                    // the lane's row has been a pivot row
  auto pivot = [&](int k) {               // column k, by its warp
    const unsigned mag = taken ? 0u : fx_mag(a) + 1u;
    const int p = __ffs(__ballot_sync(0xffffffffu, mag == __reduce_max_sync(0xffffffffu, mag))) - 1;
    const cplx v = mkc(__shfl_sync(0xffffffffu, a.x, p), __shfl_sync(0xffffffffu, a.y, p));
    const double q = 1.0 / (v.x * v.x + v.y * v.y);
    const cplx rc = mkc(v.x * q, -v.y * q);
    const cplx m = i == p ? mkc(-rc.x, -rc.y) : cmul(a, rc);
    mult[k & 1][i] = m;
    if (i == 0) s_row[k] = p;
    a = mkc(-m.x, -m.y);                  // the exchanged column
  };
  if (j == 0) pivot(0);
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const int p = s_row[k];
    if (j != k) {
      const cplx m = mult[k & 1][i];
      const cplx u = mkc(__shfl_sync(0xffffffffu, a.x, p), __shfl_sync(0xffffffffu, a.y, p));
      if (i == p) a = mkc(0.0, 0.0);
      a.x = fma(-m.x, u.x, fma(m.y, u.y, a.x));
      a.y = fma(-m.x, u.y, fma(-m.y, u.x, a.y));
    }
    taken = taken || i == p;
    if (j == k + 1 && j < n) pivot(k + 1);
    __syncthreads();
  }
  // row p_k holds unknown k, column m the coefficient of equation p_m
  if (i < n && j < n) {
    int k = 0;
    for (int q = 0; q < n; ++q)
      if (s_row[q] == i) k = q;
    X[k][s_row[j]] = a;
  }
  __syncthreads();
  if (i < n && j < n) {
    const cplx u = X[i][j], v = X[j][i];
    d.inv_out[i + n * j] = mkc(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
  }
}

}  // namespace

void launch_tikh_inv(const RegInvDesc* d, int nd, int maxn, cudaStream_t st) {
  if (nd <= 0) return;
  tikh_inv_kernel<<<nd, 32 * maxn, 0, st>>>(d);
}

// ---------------------------------------------------------------------------
// CMF2 with Gaussian modes
// ---------------------------------------------------------------------------
// D = S^-1/2 in the Cholesky form of InverseSquareRootU (maths.f90:621-644):
// S = U^H U (zpotrf 'U', column by column as the unblocked zpotf2), D = U^-1
// (ztrtri 'U','N', columns from the already inverted leading block as ztrti2),
// zeros below the diagonal; and DhS = D^H S, the matrix of A_to_B
// (cmf2_base.f90:288-292, B = (S D)^H A).  One block per (mode, set), n <= 32.
__global__ void __launch_bounds__(1024) gwp_isqrt_kernel(const GwpIsqrtDesc* __restrict__ descs, int* status) {
  const GwpIsqrtDesc& d = descs[blockIdx.x];
  const int n = d.n;
  __shared__ cplx U[MAXN_SPF][MAXN_SPF + 1];   // U[row][col]
  __shared__ cplx X[MAXN_SPF][MAXN_SPF + 1];   // U^-1
  __shared__ int bad;
  const int tid = threadIdx.x;
  if (tid == 0) bad = 0;
  for (int e = tid; e < MAXN_SPF * MAXN_SPF; e += blockDim.x) {
    const int r = e % MAXN_SPF, col = e / MAXN_SPF;
    U[r][col] = (r < n && col < n && r <= col) ? d.S[r + n * col] : mkc(0.0, 0.0);
    X[r][col] = mkc(0.0, 0.0);
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    if (tid < 32) {
      // U(j,j) = sqrt(S(j,j) - sum_{q<j} |U(q,j)|^2)
      double part = 0.0;
      for (int q = tid; q < j; q += 32) part += U[q][j].x * U[q][j].x + U[q][j].y * U[q][j].y;
      for (int off = 16; off > 0; off >>= 1) part += __shfl_down_sync(0xffffffffu, part, off);
      if (tid == 0) {
        const double ajj = U[j][j].x - part;
        if (!(ajj > 0.0)) bad = 1;
        U[j][j] = mkc(sqrt(fabs(ajj)), 0.0);
      }
    }
    __syncthreads();
    // row j right of the diagonal: (S(j,k) - sum_{q<j} conj(U(q,j)) U(q,k)) / U(j,j)
    const double rinv = 1.0 / U[j][j].x;
    for (int k = j + 1 + tid; k < n; k += blockDim.x) {
      cplx v = U[j][k];
      for (int q = 0; q < j; ++q) v = csub(v, cmul(cconj(U[q][j]), U[q][k]));
      U[j][k] = cscale(v, rinv);
    }
    __syncthreads();
  }
  for (int j = tid; j < n; j += blockDim.x) X[j][j] = mkc(1.0 / U[j][j].x, 0.0);
  __syncthreads();
  for (int j = 1; j < n; ++j) {
    // X(0:j-1, j) = -X(0:j-1, 0:j-1) U(0:j-1, j) X(j,j)
    for (int i = tid; i < j; i += blockDim.x) {
      cplx v = mkc(0.0, 0.0);
      for (int q = i; q < j; ++q) v = cadd(v, cmul(X[i][q], U[q][j]));
      X[i][j] = cscale(v, -X[j][j].x);
    }
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, col = e / n;
    d.D[e] = X[r][col];
    // (D^H S)(r, col) = sum_q conj(D(q, r)) S(q, col), S Hermitian from its upper triangle
    cplx v = mkc(0.0, 0.0);
    for (int q = 0; q <= r; ++q) {
      const cplx sq = (q <= col) ? d.S[q + n * col] : cconj(d.S[col + n * q]);
      v = cadd(v, cmul(cconj(X[q][r]), sq));
    }
    d.DhS[e] = v;
  }
  if (tid == 0 && bad) atomicOr(status, DEVST_CHOL_FAIL);
}

// Calc_DHD (hamilton.f90:535-574): same state, 1/2 (D^H (h D) + (h D)^H D) with h
// Hermitian from its upper triangle (zhemm + zher2k), real diagonal; across
// states (D1^H h) D2.  Entries of modulus <= DBL_EPSILON become zero (the
// reference's clean-up, on the upper triangle for the Hermitian case, which is
// then mirrored into the full matrix the mode products use).
__global__ void __launch_bounds__(1024) gwp_dhd_kernel(const GwpDhdDesc* __restrict__ descs) {
  const GwpDhdDesc& d = descs[blockIdx.x];
  const int n1 = d.n1, n2 = d.n2;
  __shared__ cplx aux[MAXN_SPF][MAXN_SPF + 1];
  __shared__ cplx res[MAXN_SPF][MAXN_SPF + 1];
  const int tid = threadIdx.x;
  if (d.same_state) {
    for (int e = tid; e < n1 * n2; e += blockDim.x) {   // aux = h D
      const int a = e % n1, b = e / n1;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n1; ++q) {
        const cplx hq = (a <= q) ? d.h[a + n1 * q] : cconj(d.h[q + n1 * a]);
        v = cadd(v, cmul(hq, d.D2[q + n2 * b]));
      }
      aux[a][b] = v;
    }
    __syncthreads();
    for (int e = tid; e < n1 * n2; e += blockDim.x) {
      const int a = e % n1, b = e / n1;
      if (a > b) continue;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n1; ++q) {
        v = cadd(v, cmul(cconj(d.D1[q + n1 * a]), aux[q][b]));
        v = cadd(v, cmul(cconj(aux[q][a]), d.D1[q + n1 * b]));
      }
      v = cscale(v, 0.5);
      if (a == b) v.y = 0.0;
      if (!(sqrt(v.x * v.x + v.y * v.y) > DBL_EPSILON)) v = mkc(0.0, 0.0);
      res[a][b] = v;
    }
    __syncthreads();
    for (int e = tid; e < n1 * n2; e += blockDim.x) {
      const int a = e % n1, b = e / n1;
      d.out[e] = (a <= b) ? res[a][b] : cconj(res[b][a]);
    }
  } else {
    for (int e = tid; e < n1 * n2; e += blockDim.x) {   // aux = D1^H h
      const int a = e % n1, b = e / n1;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n1; ++q) v = cadd(v, cmul(cconj(d.D1[q + n1 * a]), d.h[q + n1 * b]));
      aux[a][b] = v;
    }
    __syncthreads();
    for (int e = tid; e < n1 * n2; e += blockDim.x) {
      const int a = e % n1, b = e / n1;
      cplx v = mkc(0.0, 0.0);
      for (int q = 0; q < n2; ++q) v = cadd(v, cmul(aux[a][q], d.D2[q + n2 * b]));
      if (!(sqrt(v.x * v.x + v.y * v.y) > DBL_EPSILON)) v = mkc(0.0, 0.0);
      d.out[e] = v;
    }
  }
}

// dD = -tau D per (mode, set) block of the D vectors (cmf2_derivatives.f90:228)
__global__ void gwp_dderiv_kernel(const GwpDDerivDesc* __restrict__ descs, const cplx* __restrict__ Din,
                                  cplx* __restrict__ Dout) {
  const GwpDDerivDesc& d = descs[blockIdx.x];
  const int n = d.n;
  const cplx* D = Din + d.off;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int a = e % n, b = e / n;
    cplx v = mkc(0.0, 0.0);
    for (int q = 0; q < n; ++q) v = cadd(v, cmul(d.tau[a + n * q], D[q + n * b]));
    Dout[d.off + e] = mkc(-v.x, -v.y);
  }
}

void launch_gwp_isqrt(const GwpIsqrtDesc* d, int nd, int* status, cudaStream_t st) {
  if (nd <= 0) return;
  gwp_isqrt_kernel<<<nd, 1024, 0, st>>>(d, status);
}
void launch_gwp_dhd(const GwpDhdDesc* d, int nd, cudaStream_t st) {
  if (nd <= 0) return;
  gwp_dhd_kernel<<<nd, 1024, 0, st>>>(d);
}
void launch_gwp_dderiv(const GwpDDerivDesc* d, int nd, const cplx* Din, cplx* Dout, cudaStream_t st) {
  if (nd <= 0) return;
  gwp_dderiv_kernel<<<nd, 256, 0, st>>>(d, Din, Dout);
}

// ---------------------------------------------------------------------------
// Calc_Density (output.f90:332-445)
// ---------------------------------------------------------------------------
// GauOvl1D (gmctdh_objects.f90:1476-1493): <g1|g2> of normalised 1D Gaussians
__device__ cplx gau_ovl_1d(double a1, double a2, cplx xi1, cplx xi2) {
  const cplx s = cadd(cconj(xi1), xi2);
  cplx c = mkc(xi1.x * xi1.x / a1 + xi2.x * xi2.x / a2, 0.0);
  c = csub(c, cdivr(cmul(s, s), a1 + a2));
  const double a12 = a1 + a2;
  return cscale(cexp_(cscale(c, 0.25)), sqrt(sqrt(4.0 * a1 * a2 / (a12 * a12))));
}

__device__ __forceinline__ cplx herm_el(const cplx* X, int n, int i, int j) {
  cplx v = (i <= j) ? X[i + n * j] : cconj(X[j + n * i]);
  if (i == j) v.y = 0.0;
  return v;
}

// Grid DOF: Y_j = sum_j' rho(j, j') phi_j' (rho Hermitian from its upper
// triangle), DM(kg1, kg2) = sum_r sum_j conj(phi_j(r, kg2)) Y_j(r, kg1) with r the
// other DOFs of the mode (MatricisePsi, hamilton.f90:664-699), density = Re DM(kg, kg),
// basis populations Re sum_ab T(kg, a) DM(a, b) T(kg, b).  One block.
__global__ void __launch_bounds__(256) density_grid_kernel(DensGridArgs a) {
  const int n = a.n, nG = a.nG, ll = a.ll, nl = a.nl;
  const long long G = (long long)ll * nG * nl;
  for (long long e = threadIdx.x; e < G * n; e += blockDim.x) {
    const long long g = e % G;
    const int j = (int)(e / G);
    cplx v = mkc(0.0, 0.0);
    for (int q = 0; q < n; ++q) v = cadd(v, cmul(herm_el(a.rho, n, j, q), a.phi[g + G * q]));
    a.Y[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nG * nG; e += blockDim.x) {
    const int k1 = e % nG, k2 = e / nG;
    cplx v = mkc(0.0, 0.0);
    for (int j = 0; j < n; ++j)
      for (int ro = 0; ro < nl; ++ro)
        for (int ri = 0; ri < ll; ++ri) {
          const long long b = ri + (long long)ll * nG * ro + G * j;
          v = cadd(v, cmul(cconj(a.phi[b + (long long)ll * k2]), a.Y[b + (long long)ll * k1]));
        }
    a.DM[e] = v;
  }
  __syncthreads();
  for (int kg = threadIdx.x; kg < nG; kg += blockDim.x) {
    a.dens[kg] = a.DM[kg + nG * kg].x;
    if (a.trafo) {
      double p = 0.0;
      for (int q = 0; q < nG; ++q) {
        cplx v = mkc(0.0, 0.0);
        for (int b = 0; b < nG; ++b) v = cadd(v, cscale(a.DM[q + nG * b], a.trafo[kg + a.ldt * b]));
        p += a.trafo[kg + a.ldt * q] * v.x;
      }
      a.pop[kg] = p;
    }
  }
}

// Gaussian DOF k: density(x) = delta Re sum_{j1,j2} c(j1,j2) exp(x^2 (a1 + a2) + x (conj xi1 + xi2))
// with c = rho(j1,j2) (4/pi^2 a1 a2 exp(Re xi1^2/a1 + Re xi2^2/a2))^(1/4) times the 1D
// overlaps of the other DOFs (rho Hermitian from its upper triangle).  One block.
__global__ void __launch_bounds__(256) density_gwp_kernel(DensGwpArgs a) {
  __shared__ cplx cf[MAXN_SPF * MAXN_SPF];
  const int n = a.n, k = a.k;
  const double pi24 = 1.0 / (asin(1.0) * asin(1.0));
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int j1 = e % n, j2 = e / n;
    const double a1 = a.a[k + a.lda * j1], a2 = a.a[k + a.lda * j2];
    const cplx x1 = a.xi[k + a.nmd * j1], x2 = a.xi[k + a.nmd * j2];
    cplx c = cscale(herm_el(a.rho, n, j1, j2), pow(pi24 * a1 * a2 * exp(x1.x * x1.x / a1 + x2.x * x2.x / a2), 0.25));
    for (int q = 0; q < a.nmd; ++q) {
      if (q == k) continue;
      c = cmul(c, gau_ovl_1d(a.a[q + a.lda * j1], a.a[q + a.lda * j2], a.xi[q + a.nmd * j1], a.xi[q + a.nmd * j2]));
    }
    cf[e] = c;
  }
  __syncthreads();
  for (int kg = threadIdx.x; kg < a.nG; kg += blockDim.x) {
    const double x = a.x0 + a.delta * kg;
    double d = 0.0;
    for (int j2 = 0; j2 < n; ++j2)
      for (int j1 = 0; j1 < n; ++j1) {
        const double a12 = a.a[k + a.lda * j1] + a.a[k + a.lda * j2];
        const cplx xs = cadd(cconj(a.xi[k + a.nmd * j1]), a.xi[k + a.nmd * j2]);
        const cplx ex = cexp_(mkc(x * x * a12 + x * xs.x, x * xs.y));
        d += cmul(cf[j1 + n * j2], ex).x;
      }
    a.dens[kg] = d * a.delta;
  }
}

void launch_density_grid(const DensGridArgs& a, cudaStream_t st) { density_grid_kernel<<<1, 256, 0, st>>>(a); }
void launch_density_gwp(const DensGwpArgs& a, cudaStream_t st) { density_gwp_kernel<<<1, 256, 0, st>>>(a); }

void launch_gwp_ovl(const GwpOvlDesc* d, int nd, cudaStream_t st) {
  if (nd <= 0) return;
  gwp_ovl_kernel<<<dim3(nd, MAXN_SPF), 32, 0, st>>>(d);
}

void launch_gwp_h1(const GwpH1Desc* d, int nd, cudaStream_t st) {
  if (nd <= 0) return;
  gwp_h1_kernel<<<dim3(nd, MAXN_SPF / 2), 64, 0, st>>>(d);
}

long long gwp_y_scratch(int maxG, int maxn, int maxops) {
  return (long long)maxG * maxn * ((maxops + YOP_CHUNK - 1) / YOP_CHUNK) + (long long)maxn * maxn * maxops;
}
int launch_gwp_cy(const GwpCYDesc* d, int nd, int maxG, int maxn, int maxops, const GwpYOp* ops, cplx* part,
                  cudaStream_t st) {
  if (nd <= 0) return 0;
  const unsigned ne = (unsigned)((maxG * maxn + 255) / 256);
  gwp_sa0_kernel<<<dim3(ne, nd), 256, 0, st>>>(d);
  gwp_sa0sm1_kernel<<<dim3(ne, nd), 256, 0, st>>>(d);
  const unsigned nt = (unsigned)((maxG + 7) / 8);
  gwp_c_kernel<<<dim3(nt, nt, nd), 64, 0, st>>>(d);
  const int nch = (maxops + YOP_CHUNK - 1) / YOP_CHUNK;
  const long long g_off = (long long)maxG * maxn * nch, part_ld = gwp_y_scratch(maxG, maxn, maxops);
  const long long nthr = (long long)maxn * maxn * nch;
  if (maxops > 0) {
    gwp_y_part_kernel<<<dim3((unsigned)((nthr + 31) / 32), nd), 32, 0, st>>>(d, ops, part, part_ld, maxn);
    gwp_y_mf_kernel<<<dim3((unsigned)((maxn * maxn + 31) / 32), maxops, nd), 32, 0, st>>>(d, ops, part, part_ld, g_off);
  }
  gwp_y_sum_kernel<<<dim3(maxG, nd), 32, 0, st>>>(d, part, part_ld, g_off, maxn);
  return maxops > 0 ? 6 : 4;
}

int launch_gwp_solve(const GwpCYDesc* d, int nd, int maxG, cplx der, cplx* out, int* status, cudaStream_t st) {
  if (nd <= 0) return 0;
  const int threads = (maxG + 1 + 31) & ~31;
  int launches = 0;
  for (int j0 = 0; j0 < maxG; j0 += LU_PW) {
    lu_panel_kernel<<<nd, threads, 0, st>>>(d, j0);
    const unsigned nt = (unsigned)((maxG + 1 - j0 + 31) / 32);
    lu_update_kernel<<<dim3(nt, nt, nd), 256, 0, st>>>(d, j0);
    launches += 2;
  }
  lu_back_kernel<<<dim3(2, nd), 512, (sizeof(cplx) + sizeof(int)) * maxG, st>>>(d);
  gwp_tau_kernel<<<dim3(4, nd), 256, sizeof(cplx) * maxG, st>>>(d, der, out, status);
  return launches + 2;
}
