// Exact digit arithmetic on the FP16 tensor cores for the FP64 contractions.
// Included by spc_propagate.cu inside namespace spc.
//
// GB300 issues two FP64 FMAs per clock and SM (1.25 TFLOP/s measured over the
// chip) and 1017 FP16 products with FP32 accumulation (594 TFLOP/s measured
// for mma.sync m16n8k16). A double is therefore cut into radix-256 digits (the
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication",
// Numer. Algorithms 59 (2012)): x = sum_i d_i 256^(7-i), i = 0..7, in units
// of a common power of two, d_i in [-128, 127] (exact in FP16). Products of
// digits are at most 2^14, so sums of up to 2^10 of them are integers of at
// most 2^24 and exact in the FP32 accumulators. The product sums S_l of equal
// weight (i + j = l) are kept down to a level and closed in integers: the
// only errors are the rounding of x to the common unit (61 or 62 bits below
// the largest component), the dropped levels and the last rounding. Measured
// against extended precision they are no larger than the FP64 kernels'.
//
// The digits of a two's-complement integer v are the bytes of
// v + 0x8080808080808080, each 128 too large; a byte b becomes the FP16 number
// b - 128 as (0x6400 | b) - 1152 (0x6400 is 1024, whose unit is 1).

#define DIGITS 8
#define DIGIT_BIAS 0x8080808080808080ull

// x (sign-magnitude double) as an integer in units of 2^(E - 52 - BITS), E the
// exponent of the largest |x| of its set (biased: emax): |result| <=
// 2^(53 + BITS), rounded to nearest (half up in magnitude). Subnormals count
// as zero.
template <int BITS>
__device__ __forceinline__ long long to_fixed(double x, int emax) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)(b >> 52) & 0x7ff;
  const unsigned long long man = (b & 0xfffffffffffffll) | (1ull << 52);
  const int sh = min(emax - ex, 63);
  unsigned long long v = (((man << (BITS + 1)) >> sh) + 1) >> 1;
  v = ex == 0 ? 0 : v;
  return b < 0 ? -(long long)v : (long long)v;
}

// FP16 pair (byte k of re - 128, byte k of im - 128) from biased words
__device__ __forceinline__ unsigned digit_pair(unsigned re, unsigned im, int k) {
  const unsigned t = __byte_perm(re, im, k | ((k + 4) << 4));          // [re_k, im_k, ., .]
  const unsigned h = __byte_perm(t, 0x64646464u, 0x4140);              // 1024 + byte, twice
  const __half2 v = __hadd2(*reinterpret_cast<const __half2*>(&h), __half2half2(__ushort_as_half(0xe480)));  // - 1152
  return *reinterpret_cast<const unsigned*>(&v);
}

// D += A B, one m16n8k16 product of FP16 digits
__device__ __forceinline__ void mma_digits(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
