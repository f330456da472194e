// Exact digit arithmetic for the FP64 contractions on the tensor cores (sm_103a).
//
// GB300 issues one warp-wide FP64 instruction per SM sub-partition every 62-64
// cycles (measured 1.83 DFMA per SM and cycle, 0.53 TFMA/s on 152 SMs); its FP16
// tensor path does 1,042 multiply-adds per SM and cycle through mma.sync.  The mode
// products and contractions therefore bring their operands to a common exponent per
// short vector (a fibre, a matrix row, a tensor column) and cut the mantissas into
// signed 8-bit digits.  Digits are exact in FP16, their products and the FP32 sums
// of these are exact integers, and the sums of equal weight (digit i of one operand
// with digit k - i of the other) are joined in 64-bit integers: a product of 62-bit
// (or 54-bit) operands that rounds once, to FP64.  Narrower integer forms lose to
// this on the same kernels: 28-bit limbs in IMAD.WIDE (8 lanes per sub-partition and
// cycle) took 41 us where the digits take 26 us and FP64 takes 136 us (262,144 fibres
// of 8 x 8 complex products).
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
// the leading NS (7 or 8) digits of a (low halves) and b (high halves); dropping the
// eighth rounds to the seventh
template <int NS>
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
  if (NS > 7) s[7] = fx_half2(w3, 0x4240);
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

// sum_k D_k 2^(-8 k) 2^44 as an integer, |D_k| < 2^22, |D_0 2^44| < 2^62: the integer of D
// appears in the low bits of D + 1.5 2^23; the biases are taken out as constants.
template <int NS, int W>
__device__ __forceinline__ long long fx_join(const float (*c)[W], int i) {
  constexpr float mg = 12582912.f;
  constexpr unsigned z = 0x4B400000u, zz = (z << 8) + z;
  const float f6 = NS > 7 ? fmaf(c[NS > 7 ? 7 : 0][i], 1.f / 256.f, c[6][i]) : c[6][i];
  const unsigned F = __float_as_uint(fmaf(f6, 1.f / 16.f, mg));
  unsigned v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = __float_as_uint(c[k][i] + mg);
  const int B = (int)(v[2] * 256u + (v[3] - zz)), C = (int)(v[4] * 256u + (v[5] - (zz + z / 16u)));
  const long long t = (long long)B * 1048576 + ((long long)C * 16 + (long long)(unsigned long long)F);
  const unsigned h = (unsigned)((unsigned long long)t >> 32) + (v[0] * 4096u + v[1] * 16u) - (zz << 4);
  return (long long)(((unsigned long long)h << 32) | (unsigned)t);
}
// the same times 2^-DN, rounded, for |D_k| <= 2^24 (a conversion instruction per sum)
template <int NS, int DN>
__device__ __forceinline__ long long fx_join_wide(const float (*c)[4], int i) {
  const float f6 = NS > 7 ? fmaf(c[NS > 7 ? 7 : 0][i], 1.f / 256.f, c[6][i]) : c[6][i];
  int v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = __float2int_rn(c[k][i]);
  const long long lo = (long long)v[4] * 4096 + ((long long)v[5] * 16 + __float2int_rn(f6 * (1.f / 16.f)));
  return ((long long)(v[0] * 256 + v[1]) << (36 - DN)) + ((long long)(v[2] * 256 + v[3]) << (20 - DN)) +
         (DN ? (lo + ((1 << DN) >> 1)) >> DN : lo);
}

// The exponent, in the exponent field's place, of an integer joined to 2^bits times the
// digits' product: ea, eb the exponent words the operands were cut with.  Exponents
// below zero wrap, as unsigned words do.
__host__ __device__ __forceinline__ unsigned fx_exp(unsigned ea, unsigned eb, unsigned bits) {
  return ea + eb - ((2044u + 12u + bits) << 20);
}
__host__ __device__ __forceinline__ unsigned fx_add_exp(unsigned hi, unsigned es) { return hi ? hi + es : hi; }
// v 2^(es / 2^20) as FP64, rounded to nearest (the result is a normal number or zero).
// The conversion is one instruction of the otherwise idle FP64 pipe.
__device__ __forceinline__ double fx_double(long long v, unsigned es) {
  const double d = (double)v;
  return __hiloint2double((int)fx_add_exp((unsigned)__double2hiint(d), es), __double2loint(d));
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
