// Digit arithmetic for the FP64 contractions on the tensor cores (sm_103a).
//
// GB300 issues one warp-wide FP64 instruction per SM sub-partition every 62-64
// cycles (measured 1.83 DFMA per SM and cycle, 0.53 TFMA/s on 152 SMs); its FP16
// tensor path does 1,042 multiply-adds per SM and cycle through mma.sync.  The mode
// products and contractions therefore bring their operands to a common exponent per
// short vector (a fibre, a matrix row, a tensor column) and cut the mantissas into
// eight signed 8-bit digits (splitting operands into slices whose products are exact is
// the method of Ozaki, Ogita, Oishi and Rump, 2012).  Digits are exact in FP16, their
// products and the FP32 sums of these are exact integers, and the sums of equal weight
// (digit i of one operand with digit k - i of the other) are joined in 64-bit integers.
// Narrower integer forms lose to this on the same kernels: 28-bit limbs in IMAD.WIDE
// (8 lanes per sub-partition and cycle) took 41 us where the digits take 26 us and FP64
// takes 136 us (262,144 fibres of 8 x 8 complex products).
//
// Accuracy.  Operands are cut 62 bits below the largest element of their vector, and the
// 28 of 64 digit products of weight below 2^-64 are left out: with X and M the largest
// elements of the two vectors, a sum of n products is off by about 2^-58 X M (the dropped
// digits of n <= 16 terms, whatever their size).  An FP64 chain is off by up to
// n 2^-53 T, T = sum |x||m|.  So the digits are the more accurate where T is not far below
// X M, and every kernel sees to that: mode products and operator sums first scale the
// elements of one index by a common power of two, up in one operand and down in the other
// (weakly occupied SPFs, operators in different units), and where the sum itself (mode
// products) or a lower bound of T from one more MMA on the leading 16 bits (the others)
// stays below 2^-6 .. 2^-8 X M, it is computed again in FP64.  The bound of the FP64 chain
// then holds for all operands.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

// Exponent fields (biased) within which no intermediate leaves the normal range;
// vectors outside (and non-finite ones) take the FP64 code.
#define FX_EMIN 623
#define FX_EMAX 1423
#define FX_EBITS 0x7ff00000u

// the magnitude's leading word: orders |x| and holds the exponent field in bits 20..30
__device__ __forceinline__ unsigned fx_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ unsigned fx_mag(cplx v) { return max(fx_mag(v.x), fx_mag(v.y)); }
__device__ __forceinline__ bool fx_ok(unsigned mag) {
  return mag == 0u || (mag >= ((unsigned)FX_EMIN << 20) && mag < ((unsigned)(FX_EMAX + 1) << 20));
}
// the exponent field (in place) to cut a vector's digits with: zero vectors take the smallest
__device__ __forceinline__ unsigned fx_ebits(unsigned mag) { return max(mag & FX_EBITS, (unsigned)FX_EMIN << 20); }

// R = x 2^62 / 2^(e - 1022) for |x| < 2^(e - 1022), e the exponent field in ebits; the
// bytes of the result are R's digits (most significant first, |first| <= 64, the
// others -128 .. 127) plus 128.  Zeros and elements below the normal range are at
// least FX_EMIN binary orders below e and shift out.
__device__ __forceinline__ void fx_word(double x, unsigned ebits, unsigned& uh, unsigned& ul) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned long long t = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 9;
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(t), "r"((ebits - (hi & FX_EBITS)) >> 20));   // 0 beyond 63 bits
  const unsigned long long sg = (unsigned long long)(long long)((int)hi >> 31);
  const unsigned long long v = (r ^ sg) + (0x8080808080808080ull - sg);
  uh = (unsigned)(v >> 32);
  ul = (unsigned)v;
}
// two biased digits (bytes of w selected by sel) as signed FP16: 1024 + b - 1152
__device__ __forceinline__ unsigned fx_half2(unsigned w, unsigned sel) {
  unsigned r;
  asm("add.f16x2 %0, %1, %2;" : "=r"(r) : "r"(__byte_perm(w, 0x64646464u, sel)), "r"(0xE480E480u));
  return r;
}
// the digits of a (low halves) and b (high halves)
#define FX_NS 8
__device__ __forceinline__ void fx_digits(double a, double b, unsigned ea, unsigned eb, unsigned* s) {
  unsigned ah, al, bh, bl;
  fx_word(a, ea, ah, al);
  fx_word(b, eb, bh, bl);
  const unsigned w0 = __byte_perm(ah, bh, 0x7632), w1 = __byte_perm(ah, bh, 0x5410);
  const unsigned w2 = __byte_perm(al, bl, 0x7632), w3 = __byte_perm(al, bl, 0x5410);
  s[0] = fx_half2(w0, 0x4341);
  s[1] = fx_half2(w0, 0x4240);
  s[2] = fx_half2(w1, 0x4341);
  s[3] = fx_half2(w1, 0x4240);
  s[4] = fx_half2(w2, 0x4341);
  s[5] = fx_half2(w2, 0x4240);
  s[6] = fx_half2(w3, 0x4341);
  s[7] = fx_half2(w3, 0x4240);
}

// C (+)= A B on the tensor cores, A 16 x 16 (or 16 x 8) row-major, B 16 x 8 columns, FP16
// operands, FP32 sums; `first` starts from zero
__device__ __forceinline__ void fx_mma16(float* c, const unsigned* a, unsigned b0, unsigned b1, bool first) {
  if (first)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void fx_mma8(float* c, const unsigned* a, unsigned b0, bool first) {
  if (first)
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5},{%6},{%7,%7,%7,%7};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(b0), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5},{%6},{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(b0));
}

// sum_k D_k 2^(-8 k) 2^(44 + sh) of eight sums as an integer, |D_k 2^sh| < 2^22 and the
// result below 2^62: the integer of D appears in the low bits of D + 1.5 2^23; the biases
// are taken out as constants.  pw = 2^sh.
template <int W>
__device__ __forceinline__ long long fx_join(const float (*c)[W], int i, float pw) {
  constexpr float mg = 12582912.f;
  constexpr unsigned z = 0x4B400000u, zz = (z << 8) + z;
  const float f6 = fmaf(c[7][i], 1.f / 256.f, c[6][i]);
  const unsigned F = __float_as_uint(fmaf(f6, pw * (1.f / 16.f), mg));
  unsigned v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = __float_as_uint(fmaf(c[k][i], pw, mg));
  const int B = (int)(v[2] * 256u + (v[3] - zz)), C = (int)(v[4] * 256u + (v[5] - (zz + z / 16u)));
  const long long t = (long long)B * 1048576 + ((long long)C * 16 + (long long)(unsigned long long)F);
  const unsigned h = (unsigned)((unsigned long long)t >> 32) + (v[0] * 4096u + v[1] * 16u) - (zz << 4);
  return (long long)(((unsigned long long)h << 32) | (unsigned)t);
}
// the bits that a sum of n complex terms leaves for it; by the sum's own terms, not by the
// launch's largest, so that a product is the same in every batch
__host__ __device__ constexpr int fx_headroom(int n) {
  return n <= 1 ? 4 : (n <= 2 ? 3 : (n <= 4 ? 2 : (n <= 8 ? 1 : 0)));
}
__device__ __forceinline__ float fx_pow2(int sh) { return __uint_as_float((unsigned)(127 + sh) << 23); }
// the same for |D_k 2^sh| <= 2^24 (a conversion instruction per sum)
__device__ __forceinline__ long long fx_join_wide(const float (*c)[4], int i, float pw) {
  const float f6 = fmaf(c[7][i], 1.f / 256.f, c[6][i]);
  int v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = __float2int_rn(c[k][i] * pw);
  const long long lo = (long long)v[4] * 4096 + ((long long)v[5] * 16 + __float2int_rn(f6 * (pw * (1.f / 16.f))));
  return ((long long)(v[0] * 256 + v[1]) << 36) + ((long long)(v[2] * 256 + v[3]) << 20) + lo;
}
// All of it, of the sums a[.][i] + b[.][j] (or -, |D_k| <= 2^24 each): sum_k<4 D_k 2^(24 - 8 k)
// and sum_k>=4 D_k 2^(56 - 8 k), both below 2^53.
template <bool SUB>
__device__ __forceinline__ void fx_join_pair(const float (*a)[4], int i, const float (*b)[4], int j, long long& hi,
                                             long long& lo) {
  auto D = [&](int k) {
    const int u = __float2int_rn(a[k][i]), v = __float2int_rn(b[k][j]);
    return SUB ? u - v : u + v;
  };
  hi = (long long)D(0) << 24;
  hi += (long long)D(1) << 16;
  hi += (long long)D(2) * 256 + D(3);
  lo = (long long)D(4) << 24;
  lo += (long long)D(5) << 16;
  lo += (long long)D(6) * 256 + D(7);
}
// Both components below 2^-7 .. 2^-9 of the product of the largest operands (which is
// between 2^(54 + sh) and 2^(56 + sh) in the units of fx_join), where the rounding of
// fx_join, half a unit, passes the n 2^-52 of an FP64 chain: T = sum |x||m| decides.
// limit: fx_small_limit(sh), or 0 for fibres of zeros.
__device__ __forceinline__ unsigned fx_small_limit(int sh) { return 32768u << sh; }
__device__ __forceinline__ unsigned fx_small_word(long long re, long long im, unsigned limit) {
  return ((unsigned)(re >> 32) + limit) | ((unsigned)(im >> 32) + limit);
}
__device__ __forceinline__ bool fx_small(long long re, long long im, unsigned limit) {
  return fx_small_word(re, im, limit) < 2 * limit;
}
// ... T of the leading digits (fx_lead) below the same, the largest operands' product being
// 2^26 .. 2^28; (|xr| + |xi|)(|mr| + |mi|) is up to twice |x||m|
#define FX_LOW 1048576.f
// |x| of the two leading digits, in units of 2^-14 of 2^(e - 1022) (FP16, 11 bits of it)
__device__ __forceinline__ unsigned fx_lead(unsigned s0, unsigned s1) {
  unsigned r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(s0), "r"(0x5C005C00u), "r"(s1));
  return r & 0x7fff7fffu;
}
__device__ __forceinline__ unsigned fx_add_half2(unsigned a, unsigned b) {
  unsigned r;
  asm("add.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// its two halves, (re, im), added
__device__ __forceinline__ float fx_lead_sum(unsigned s0, unsigned s1) {
  const unsigned l = fx_lead(s0, s1);
  float f;
  asm("{\n\t.reg .b16 h, g;\n\tmov.b32 {h, g}, %1;\n\tcvt.f32.f16 %0, h;\n\t}" : "=f"(f)
      : "r"(fx_add_half2(l, __byte_perm(l, l, 0x1032))));
  return f;
}

// The exponent, in the exponent field's place, of an integer joined to 2^bits times the
// digits' product: ea, eb the exponent words the operands were cut with.  Exponents
// below zero wrap, as unsigned words do.
__host__ __device__ __forceinline__ unsigned fx_exp(unsigned ea, unsigned eb, unsigned bits) {
  return ea + eb - ((2044u + 12u + bits) << 20);
}
__host__ __device__ __forceinline__ unsigned fx_add_exp(unsigned hi, unsigned es) { return hi ? hi + es : hi; }
// fx_join_pair's sum as FP64; es with bits = 24
__device__ __forceinline__ double fx_double_pair(long long hi, long long lo, unsigned es);
// v 2^(es / 2^20) as FP64, rounded to nearest (the result is a normal number or zero).
// The conversion is one instruction of the otherwise idle FP64 pipe.
__device__ __forceinline__ double fx_double(long long v, unsigned es) {
  const double d = (double)v;
  return __hiloint2double((int)fx_add_exp((unsigned)__double2hiint(d), es), __double2loint(d));
}
__device__ __forceinline__ double fx_double_pair(long long hi, long long lo, unsigned es) {
  return fx_double(hi, es) + fx_double(lo, es - (32u << 20));   // both exact: below 2^53
}

// A mode product's fibre (l, :, r) in FP64, for fibres or matrices outside the exponent range.
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

// Outputs first + step i of fibre p for the bits i of `mask`, in FP64.
static __device__ __noinline__ void prod_outputs_fp64(const ProdDesc& d, unsigned p, unsigned mask, int first, int step) {
  const long long L = d.L, r = p / L;
  const cplx* x = d.X + (p + L * (d.nin - 1) * r);
  for (; mask; mask &= mask - 1) {
    const int jo = first + step * (__ffs(mask) - 1);
    const cplx* m = d.M + (d.conjT ? (long long)d.ldm * jo : jo);
    const long long sm = d.conjT ? 1 : d.ldm;
    cplx v[4] = {mkc(0.0, 0.0), mkc(0.0, 0.0), mkc(0.0, 0.0), mkc(0.0, 0.0)};   // four chains, eight loads in flight
    for (int j = 0; j < d.nin; j += 4) {
      cplx a[4], b[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        a[k] = j + k < d.nin ? m[sm * (j + k)] : mkc(0.0, 0.0);
        b[k] = j + k < d.nin ? x[L * (j + k)] : mkc(0.0, 0.0);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) cfma(v[k], d.conjT ? cconj(a[k]) : a[k], b[k]);
    }
    const cplx s = cmul(d.alpha, cadd(cadd(v[0], v[1]), cadd(v[2], v[3])));
    cplx* y = d.Y + (p + L * (d.nout - 1) * r) + L * jo;
    *y = d.accumulate ? cadd(s, *y) : s;
  }
}

// The scaling of a mode product's input index: element j of the fibres times 2^b(j), the
// matrix's column j times 2^-b(j), so that the tensor's columns are alike in size whatever
// the SPFs' occupations.  Column sizes (colmag[j], exponent words) are the mean exponents
// over FX_SAMPLE fibres spread over the tensor, the same for every CTA and kernel: any
// powers of two are right, and fibres that these do not suit show in the sums (from the
// largest elements, which one fibre decides, ten times as many).  Empty columns count
// as the weakest; columns within 2^FX_SCALE_MIN of each other are left alone,
// as a sample's mean is no better than that.  In exponent words; lane j returns b(j).
#define FX_SCALE_MAX 60
#define FX_SCALE_MIN 1
#define FX_SAMPLE 32
// the sizes of the columns of the sample, a warp per column in turn
__device__ __forceinline__ void fx_column_sizes(const ProdDesc& d, unsigned* colmag) {
  const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const unsigned L = (unsigned)d.L, nfib = (unsigned)(d.L * d.R);
  const unsigned p = (unsigned)((unsigned long long)nfib * lane / FX_SAMPLE);
  const cplx* x = d.X + (p + (long long)L * (d.nin - 1) * (p / L));
#pragma unroll 4
  for (int j = threadIdx.x >> 5; j < d.nin; j += nwarp) {
    const unsigned m = fx_mag(x[(long long)L * j]), some = __ballot_sync(0xffffffffu, m);
    const unsigned sum = __reduce_add_sync(0xffffffffu, m >> 20);
    if (lane == 0) colmag[j] = some ? max(sum / __popc(some), 1u) << 20 : 0u;
  }
}
// x 2^b; what is above or below the normal range stays (it fails fx_ok, or is below every digit)
__device__ __forceinline__ double fx_scale_up(double x, unsigned b) {
  const unsigned hi = (unsigned)__double2hiint(x), e = hi & FX_EBITS;
  return __hiloint2double((int)(e - 1u < (1500u << 20) ? hi + b : hi), __double2loint(x));
}
__device__ __forceinline__ cplx fx_scale_up(cplx x, unsigned b) { return mkc(fx_scale_up(x.x, b), fx_scale_up(x.y, b)); }
// the magnitude word of m 2^-b: zeros stay zero, and what leaves the range fails fx_ok
__device__ __forceinline__ unsigned fx_scaled_down(unsigned mag, unsigned b) { return mag ? (mag > b ? mag - b : 1u) : 0u; }
__device__ __forceinline__ unsigned fx_column_scale(const unsigned* colmag, int n) {
  const int lane = threadIdx.x & 31;
  const unsigned m = lane < n ? colmag[lane] : 0u;
  const unsigned top = __reduce_max_sync(0xffffffffu, m) & FX_EBITS;
  const unsigned low = __reduce_min_sync(0xffffffffu, m ? m : 0xffffffffu);
  const unsigned own = (m ? m : min(low, top)) & FX_EBITS;
  if (top - (min(low, top) & FX_EBITS) <= (unsigned)FX_SCALE_MIN << 20) return 0u;
  return lane < n ? min(top - own, (unsigned)FX_SCALE_MAX << 20) : 0u;
}

// Descriptor of block b, found by every warp for itself: 32 candidates per round
// (descriptors are sorted by block_start).
template <typename D>
__device__ __forceinline__ int warp_find_desc(const D* __restrict__ descs, int ndesc, long long b) {
  const int lane = threadIdx.x & 31;
  int lo = 0, n = ndesc;
  while (n > 1) {
    const int step = (n + 31) >> 5;
    const int i = lo + lane * step;
    const bool le = (lane * step < n) && descs[i].block_start <= b;
    const int k = __popc(__ballot_sync(0xffffffffu, le)) - 1;   // block_start of the first is never above b
    lo += k * step;
    n = min(step, n - k * step);
  }
  return lo;
}
