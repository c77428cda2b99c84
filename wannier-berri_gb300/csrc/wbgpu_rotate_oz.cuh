// Band-basis rotation Xbar = U^dagger X U in FP64 (and double-float) accuracy on the fp16 tensor
// cores: the operands are cut into 8-bit slices whose products the tensor cores sum exactly.
// Included by wbgpu_rotate_tc.cu inside its namespace (shared tcgen05 / mbarrier helpers).
//
// The scheme is Ozaki's (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59, 2012): slices
// short enough that their products sum without rounding.
//
// Every operand is brought to 64-bit fixed point relative to the largest exponent of its vector along the
// contraction -- a row of X, a column of U, a column of T = X U (whose rows enter with the exponents of the
// rows of X) --, v with |v| < 2^62, and written as signed digits v = sum_i d_i 2^(56 - 8 i), d_i in [-128, 127]:
// the bytes of v + 0x8080..80, less 128 each.  A digit is an exact fp16 number, a product of two
// an integer below 2^14, and the products of one significance g = i + j, summed over K <= 256 and
// the pairs of a group, stay below 2^24 (up to K = 128; beyond, that is above nw = 64, only the groups g >= 4
// could pass it, whose last unit is 2^-44 of the result): FP32 accumulation in tensor memory is exact.  The NG
// groups g < NG are kept (8 for FP64: 36 pairs; 7 for double-float: 28) and recombined in 64-bit
// integers: sum_g acc_g 2^(8 (NG - 1 - g)).  The dropped pairs lie 2^-58 (FP64) and 2^-50
// (double-float) below the product of the two vectors' largest elements, so each GEMM rounds once, like an FP64 sum
// of exact products.  What that floor leaves open, next to FP64 products of every element: a sum in which
// the large elements of a row of X meet only elements of U below 2^-9 of their column's largest.  Subnormals
// count as zero.
// Error against 113-bit products, 2-norm, random X and unitary U: 4.9e-17 at nw = 32 and 5.5e-17 at nw = 128, with
// elements of X spread over e^+-16 5.4e-17 and 8.2e-17; the CUDA-core FP64 chains gave 3.8e-16, 7.6e-16, 4e-16 and
// 6e-16.  One scale per matrix gave 1.3e-15 in the last case and lost small blocks next to large ones.
//
// Bound by the CUDA cores: cutting the operands (about 40 instructions an element), recombining
// the groups and the conversions run on integer units, since the FP64 pipe (64 times slower than FP32)
// is what this avoids.  nw = 32, 9 fields, 13 824 k-points: 44.8 ms (CUDA-core FP64, 97% of the pipe)
// -> 5.9 ms (as with one scale per matrix; T goes to its columns through shared memory, so that a thread finds most
// of a column's exponent by itself and writes its digits in 16-byte pieces: from the rows' side, with warp
// reductions, 6.6 ms).  nw = 8, 110 592 k-points: 3.1 ms (2.9 with one scale).  nw = 96, 9 fields, 512 k-points:
// 27.7 ms (double-float) -> 3.8 ms, 53.4 ms (FP64) -> 4.0 ms.
//
// Complex products are embedded in real ones as in the TF32 kernel above; operand rows are 128-byte
// (64-byte) swizzled K-major rows of 64 (32) fp16.  Consecutive B slices are consecutive rows of
// shared memory and their products consecutive accumulators, so one tcgen05.mma of N = up to 256
// multiplies A slice i by several B slices: A is read from shared memory once per 256 columns.

constexpr int OZ_FMAX = 256;  // fields of one launch (their selection is kept in shared memory)

template <int DF> struct OzCfg;  // 0: complex128 in and out; 1: double-float complex in, complex64 out
template <> struct OzCfg<0> {
  typedef double2 VI;
  typedef double2 VO;
  typedef double PI;  // one part (re or im) of VI
  static constexpr int NG = 8, BIAS = 1084, EMAX = 0x7ff;
};
template <> struct OzCfg<1> {
  typedef float4 VI;  // re.hi, re.lo, im.hi, im.lo
  typedef float2 VO;
  typedef float2 PI;
  static constexpr int NG = 7, BIAS = 188, EMAX = 0xff;
};

// Biased exponents and fixed point of one real number: x = v 2^(emax - BIAS), |v| < 2^62
WBG_D int oz_exp(double x) { return (int)((unsigned)__double2hiint(x) >> 20) & 0x7ff; }
WBG_D int oz_exp(float x) { return (int)(__float_as_uint(x) >> 23) & 0xff; }
WBG_D long long oz_fix(double x, int emax) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(u >> 52) & 0x7ff;
  const int s = emax - e;
  if (e == 0 || s > 62) return 0;  // zero, subnormal, or below the last digit
  const long long v = (long long)((((u & 0xfffffffffffffull) | 0x10000000000000ull) << 9) >> s);
  return (long long)u < 0 ? -v : v;
}
WBG_D long long oz_fix(float x, int emax) {
  const uint32_t u = __float_as_uint(x);
  const int e = (int)(u >> 23) & 0xff;
  const int s = emax - e;
  if (e == 0 || s > 62) return 0;
  const long long v = (long long)(((unsigned long long)((u & 0x7fffffu) | 0x800000u) << 38) >> s);
  return (int)u < 0 ? -v : v;
}
// the same of the low half of a double-float: the multiplication by 2^(BIAS - emax), exact in two steps, and a
// truncating conversion.  It runs on the FP64 pipe, which is idle here: nw = 82 as below takes 15.2 ms with both
// halves on the integer pipe, 15.9 ms with both here, 14.7 ms with one on each.
WBG_D long long oz_fix_lo(float x, int emax) {
  const int t = 188 - emax, ta = t / 2;
  return __float2ll_rz(x * __int_as_float((ta + 127) << 23) * __int_as_float((t - ta + 127) << 23));
}
WBG_D int oz_cexp(double2 a) { return max(oz_exp(a.x), oz_exp(a.y)); }
WBG_D int oz_cexp(float4 a) { return max(oz_exp(a.x), oz_exp(a.z)); }
WBG_D long long oz_re(double2 a, int emax) { return oz_fix(a.x, emax); }
WBG_D long long oz_im(double2 a, int emax) { return oz_fix(a.y, emax); }
WBG_D long long oz_part(double a, int emax) { return oz_fix(a, emax); }
WBG_D long long oz_part(float2 a, int emax) { return oz_fix(a.x, emax) + oz_fix_lo(a.y, emax); }
WBG_D double oz_zero(double) { return 0.0; }
WBG_D float2 oz_zero(float2) { return make_float2(0.f, 0.f); }
WBG_D double2 oz_zero(double2) { return make_double2(0.0, 0.0); }
WBG_D double2 oz_real(double2 a) { return make_double2(a.x, 0.0); }
WBG_D float4 oz_real(float4 a) { return make_float4(a.x, a.y, 0.f, 0.f); }

// q 2^E rounded to nearest even, in integer arithmetic (the FP64 pipe converts 64 times slower)
WBG_D double oz_to_double(long long q, int E) {
  if (q == 0) return 0.0;
  const unsigned long long a = q < 0 ? 0ull - (unsigned long long)q : (unsigned long long)q;
  const int lz = __clzll((long long)a);
  const unsigned long long m = a << lz;
  unsigned long long r = m >> 11;
  const unsigned rem = (unsigned)m & 0x7ffu;
  r += (rem + ((unsigned)r & 1u)) > 0x400u ? 1u : 0u;
  const int be = E - lz + 11 + 52 + 1023;  // biased exponent
  unsigned long long bits;
  if (be <= 0) bits = 0;                                    // below the normal range
  else if (be >= 2047) bits = 0x7ff0000000000000ull;
  else bits = ((unsigned long long)(be - 1) << 52) + r;     // r's leading bit adds the one
  return __longlong_as_double((long long)(bits | (q < 0 ? 0x8000000000000000ull : 0ull)));
}
WBG_D float oz_to_float(long long q, int E) {
  const float f = __ll2float_rn(q);
  const int a = max(-126, min(127, E / 2)), b = max(-126, min(127, E - a));  // two exact steps
  return f * __uint_as_float((uint32_t)(a + 127) << 23) * __uint_as_float((uint32_t)(b + 127) << 23);
}
WBG_D double2 oz_pack(double2, long long re, long long im, int E) {
  return make_double2(oz_to_double(re, E), oz_to_double(im, E));
}
WBG_D float2 oz_pack(float2, long long re, long long im, int E) {
  return make_float2(oz_to_float(re, E), oz_to_float(im, E));
}
WBG_D double2 oz_nan(double2) { const double q = __longlong_as_double(0x7ff8000000000000ll); return make_double2(q, q); }
WBG_D float2 oz_nan(float2) { const float q = __int_as_float(0x7fc00000); return make_float2(q, q); }

// Digits of byte `idx` (3 most significant) of two biased words as fp16 pair: 1024 + byte - 1152
WBG_D uint32_t oz_dig2(uint32_t a, uint32_t b, int idx) {
  const uint32_t sel = (uint32_t)idx * 0x0011u | (uint32_t)(4 + idx) * 0x1100u;
  const uint32_t p = (__byte_perm(a, b, sel) & 0x00ff00ffu) | 0x64006400u;
  const uint32_t c = 0x64806480u;
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&p), *reinterpret_cast<const __half2*>(&c));
  return *reinterpret_cast<const uint32_t*>(&d);
}
WBG_D unsigned long long oz_bias(long long v) { return (unsigned long long)v + 0x8080808080808080ull; }
WBG_D uint32_t oz_word(unsigned long long w, int slice) { return slice < 4 ? (uint32_t)(w >> 32) : (uint32_t)w; }

// Byte offset of the 16-byte chunk c (8 fp16 along K) of operand row r (2 KP bytes, swizzled)
template <int KP> WBG_D uint32_t oz_off(int r, int c) {
  if (KP == 64) return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));
  if (KP == 32) return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
  return (uint32_t)(r * 32 + ((c ^ ((r >> 2) & 1)) << 4));
}
// Shared-memory descriptor of a swizzled K-major operand: SBO = 8 rows, version 1, swizzle 128 / 64 / 32 B
template <int KP> WBG_D uint64_t oz_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | (1ull << 16) | ((uint64_t)(8 * KP * 2 / 16) << 32) | (1ull << 46) |
         ((KP == 64 ? 2ull : KP == 32 ? 4ull : 6ull) << 61);
}
WBG_D void mma_f16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// Every slice product with i + j < NG of one K chunk: accumulators g at d + g ncol.
template <int KP, int NG>
WBG_D void oz_issue(uint32_t d, uint32_t a, uint32_t b, int ncol, int ksteps, uint32_t accumulate) {
  const uint32_t astride = 128 * KP * 2, bstride = (uint32_t)ncol * KP * 2;
  const int per = 256 / ncol;  // B slices per instruction
  for (int ks = 0; ks < ksteps; ++ks) {
    for (int i = 0; i < NG; ++i) {
      for (int j = 0; j < NG - i; j += per) {
        const int n = min(per, NG - i - j) * ncol;
        // D f32 (bits 4-5 = 1), A and B f16, both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
        mma_f16(d + (uint32_t)((i + j) * ncol), oz_desc<KP>(a + i * astride + ks * 32),
                oz_desc<KP>(b + j * bstride + ks * 32), idesc, accumulate | (uint32_t)(ks > 0 || i > 0));
      }
    }
  }
}

// The same with the loops unrolled (NCOL columns a slice, all K steps): a few instructions a product
template <int KP, int NG, int NCOL>
WBG_D void oz_issue_all(uint32_t d, uint32_t a, uint32_t b, uint32_t accumulate) {
  constexpr uint32_t astride = 128 * KP * 2, bstride = NCOL * KP * 2;
  constexpr int per = 256 / NCOL;
  const uint64_t ad = oz_desc<KP>(a), bd = oz_desc<KP>(b);
#pragma unroll
  for (int ks = 0; ks < KP / 16; ++ks)
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int j = 0; j < NG - i; j += per) {
        const int n = (per < NG - i - j ? per : NG - i - j) * NCOL;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
        mma_f16(d + (uint32_t)((i + j) * NCOL), ad + ((i * astride + ks * 32) >> 4), bd + ((j * bstride + ks * 32) >> 4),
                idesc, ks > 0 || i > 0 ? 1u : accumulate);
      }
}

// 8 fixed-point values along K as one 16-byte chunk of each of NS slices
template <int NS> WBG_D void oz_put8(unsigned char* base, uint32_t stride, uint32_t off, const long long (&v)[8]) {
  unsigned long long w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] = oz_bias(v[q]);
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    uint4 o;
    o.x = oz_dig2(oz_word(w[0], i), oz_word(w[1], i), 3 - (i & 3));
    o.y = oz_dig2(oz_word(w[2], i), oz_word(w[3], i), 3 - (i & 3));
    o.z = oz_dig2(oz_word(w[4], i), oz_word(w[5], i), 3 - (i & 3));
    o.w = oz_dig2(oz_word(w[6], i), oz_word(w[7], i), 3 - (i & 3));
    *reinterpret_cast<uint4*>(base + i * stride + off) = o;
  }
}
// 4 values along K (half a chunk) to two places, the second one with the sign `flip` applied
template <int NS>
WBG_D void oz_put4x2(unsigned char* base, uint32_t stride, uint32_t off0, uint32_t off1, uint32_t flip,
                     const long long (&v)[4]) {
  unsigned long long w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) w[q] = oz_bias(v[q]);
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    uint2 o;
    o.x = oz_dig2(oz_word(w[0], i), oz_word(w[1], i), 3 - (i & 3));
    o.y = oz_dig2(oz_word(w[2], i), oz_word(w[3], i), 3 - (i & 3));
    *reinterpret_cast<uint2*>(base + i * stride + off0) = o;
    *reinterpret_cast<uint2*>(base + i * stride + off1) = make_uint2(o.x ^ flip, o.y ^ flip);
  }
}

// 2 values along K (a quarter chunk) to two places, the second one with the sign `flip` applied
template <int NS>
WBG_D void oz_put2x2(unsigned char* base, uint32_t stride, uint32_t off0, uint32_t off1, uint32_t flip, long long a,
                     long long b) {
  const unsigned long long wa = oz_bias(a), wb = oz_bias(b);
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const uint32_t d = oz_dig2(oz_word(wa, i), oz_word(wb, i), 3 - (i & 3));
    *reinterpret_cast<uint32_t*>(base + i * stride + off0) = d;
    *reinterpret_cast<uint32_t*>(base + i * stride + off1) = d ^ flip;
  }
}

WBG_D void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
// exact integer of an accumulator: |x| <= 2^22 by one addition (its low bits then hold the integer),
// any |x| < 2^24 by the conversion unit, which runs at a quarter of the rate
WBG_D int oz_int_small(uint32_t r) { return __float_as_int(__uint_as_float(r) + 12582912.f) - 0x4B400000; }
WBG_D int oz_int(uint32_t r) { return __float2int_rn(__uint_as_float(r)); }
// 4 result columns of this thread's row: sum_g acc_g 2^(8 (NG - 1 - g)) >> sh, rounded.  KMAX bounds
// the contraction: group g sums at most g + 1 pairs, two of them with a leading digit (<= 64).
template <int NG, int KMAX> WBG_D void oz_cols4(uint32_t taddr, int ncol, int sh, long long* q) {
  uint32_t r[NG][4];
#pragma unroll
  for (int g = 0; g < NG; ++g) tmem_ld4(taddr + (uint32_t)(g * ncol), r[g]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int g = 0; g < NG; ++g) asm volatile("" : "+r"(r[g][0]), "+r"(r[g][1]), "+r"(r[g][2]), "+r"(r[g][3])::"memory");
  constexpr int W = 8 * (NG - 4);  // bits below hi
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    long long hi, lo;
    if (KMAX <= 64) {  // |acc_0..3| < 2^22, every pair below fits 32 bits
      const int t1 = oz_int_small(r[0][c]) * 256 + oz_int_small(r[1][c]);
      const int t2 = oz_int_small(r[2][c]) * 256 + oz_int_small(r[3][c]);
      const int t3 = oz_int(r[4][c]) * 256 + oz_int(r[5][c]);
      hi = (long long)t1 * 65536 + t2;
      if (NG == 8) lo = (long long)t3 * 65536 + (oz_int(r[6][c]) * 256 + oz_int(r[NG - 1][c]));
      else lo = (long long)t3 * 256 + oz_int(r[6][c]);
    } else {
      const int t1 = oz_int_small(r[0][c]) * 256 + oz_int_small(r[1][c]);
      hi = (long long)t1 * 65536 + ((long long)oz_int(r[2][c]) * 256 + oz_int(r[3][c]));
      lo = (long long)oz_int(r[4][c]) * 256 + oz_int(r[5][c]);
      if (NG == 8) lo = lo * 65536 + ((long long)oz_int(r[6][c]) * 256 + oz_int(r[NG - 1][c]));
      else lo = lo * 256 + oz_int(r[6][c]);
    }
    q[c] = (hi << (W - sh)) + ((lo + (1ll << (sh - 1))) >> sh);
  }
}

// Exponent of a value q 2^ex for the scale of its column: |q| < 2^bits with bits >= 32 (a smaller q is an
// integer all the same, and loses nothing at this scale), 0 of q = 0
WBG_D int oz_top(long long q, int ex) {
  const int h = (int)(q >> 32);
  return q != 0 ? ex + 64 - __clz(h ^ (h >> 31)) : 0;
}
// q 2^s (s < 63), the fraction cut off (floor)
WBG_D long long oz_shift(long long q, int s) { return s >= 0 ? q << min(s, 62) : q >> min(-s, 63); }
WBG_D int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// ---------------------------------------------------------------------------------------
// nw <= 32: the fields of one k-point stack along M as in rotate_tc_kernel (FPT fields of nw rows
// in a 128-row tile), both GEMMs share the embedded U.  KP = 16 (nw <= 8), 32 (nw <= 16) or 64 fp16
// of K; 8 KP threads a CTA and 64 / KP CTAs an SM (512 tensor memory columns in all).
// ---------------------------------------------------------------------------------------
constexpr int OZ_LDQ = 129;  // 64-bit words from a column of T to the next: its readers fall on distinct banks
template <int KP> constexpr int oz_small_smem() { return 8 * 128 * KP * 2 + 8 * KP * KP * 2 + 1024; }

template <int KP>
__global__ void __launch_bounds__(8 * KP, 64 / KP)
    rotate_oz_small(const double2* __restrict__ U, long long strideU, const double2* __restrict__ X, int nFin,
                    const int* __restrict__ fsel, const int* __restrict__ herm, int nFrot, double2* __restrict__ Xbar,
                    int nw, int nk, int fpt, int ntiles, int ldf) {
  typedef OzCfg<0> Cfg;
  constexpr int NG = Cfg::NG, THR = 8 * KP, NCG = THR / 128;
  constexpr int SH = KP == 64 ? 12 : KP == 32 ? 11 : 10;  // K <= KP: |sum| <= 2^(68 + log2 KP)
  constexpr int EP = SH + 112 - 8 * (NG - 1);
  constexpr uint32_t ASTR = 128 * KP * 2;
  constexpr uint32_t COLS = 8 * KP;
  extern __shared__ __align__(1024) unsigned char smo[];
  unsigned char* As = smo + ((1024u - (smem_u32(smo) & 1023u)) & 1023u);
  unsigned char* Bs = As + NG * ASTR;
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s, ubad_s;
  __shared__ int code_s[OZ_FMAX];  // per field: -1 invalid selection, else source | herm << 28
  // largest exponents: of each column of U, of each row (field, m) of X, of each column (field, n) of T (exponent of
  // the row of X + bits, 0: the column is zero); fields with a non-finite element
  __shared__ int ue_s[32], xe_s[128], te_s[128], fbad_s[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t mb = smem_u32(&mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_s = 0;
    ubad_s = 0;
  }
  if (tid < 128) {
    xe_s[tid] = 1;
    te_s[tid] = 0;
  }
  if (tid < 32) {
    ue_s[tid] = 1;
    fbad_s[tid] = 0;
  }
  for (int f = tid; f < nFrot; f += THR) {
    const int fs = fsel[f];
    code_s[f] = fs >= 0 && fs < nFin ? fs | (herm[f] & 7) << 28 : -1;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  const int nwp = (nw + 7) & ~7, ncol = 2 * nwp, cpr = nwp / 8, nw2 = nw * nw;
  const int quarter = warp & 3;
  const int row = 32 * quarter + lane;  // operand / accumulator row of this thread
  const int ncg = ncol / NCG;           // accumulator columns of this thread: c0 .. c0 + ncg - 1
  const int c0 = (warp >> 2) * ncg;
  const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
  const uint32_t bstr = (uint32_t)ncol * KP * 2;
  const int ldst = nwp + 1;  // staging: [row][m'] re plane, then im plane
  long long* stre = reinterpret_cast<long long*>(As);
  long long* stim = stre + 128 * ldst;
  long long* tq = stre;  // between the GEMMs: T, [column][row]
  const unsigned long long wait_ns = g_tc_wait_ns;
  uint32_t phase = 0;
  // task of the X loads: 8 columns n0.. of row r; 8 lanes take 8 rows (16-byte stores: no conflicts).
  // The values stay as loaded until their use, so that a prefetch does not wait for them.
  const int xrow = (tid / (8 * cpr)) * 8 + (tid & 7), xc8 = (tid >> 3) % cpr;
  const int xfl = xrow / nw, xm = xrow - xfl * nw;
  const uint32_t magic = 0xffffffffu / (uint32_t)nw + 1;  // r / nw = umulhi(r, magic) for r nw < 2^32
  double2 xr[8];
  auto load_x = [&](long long k, int t) {
    const int f0 = t * fpt, rows = min(fpt, nFrot - f0) * nw;
    const int code = xrow < rows ? code_s[f0 + xfl] : -1;
    const double2* src = X + (k * nFin + (code & 0xfffffff)) * (long long)nw2;
    const bool lower = (code >> 30) & 1;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int n = 8 * xc8 + c;
      xr[c] = code >= 0 && n < nw ? src[lower && n > xm ? n * nw + xm : xm * nw + n] : make_double2(0.0, 0.0);
    }
  };
  if (blockIdx.x < nk) load_x(blockIdx.x, 0);
  for (long long k = blockIdx.x; k < nk && !abort_s; k += gridDim.x) {
    // ---- embedded U_k (B operand): 4 rows j of one column n per thread
    const double2* Uk = U + k * strideU;
    {
      const int n = tid % nwp, j0 = (tid / nwp) * 4;
      double2 u[4];
      int e = 1;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const bool ok = n < nw && j0 + c < nw;
        u[c] = ok ? Uk[(j0 + c) * nw + n] : make_double2(0.0, 0.0);
        e = max(e, oz_cexp(u[c]));
      }
      if (j0 < nw) atomicMax(&ue_s[n], e);
      if (e >= Cfg::EMAX) ubad_s = 1;
      __syncthreads();
      if (j0 < nwp) {
        const int eu = ue_s[n];
        long long v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = oz_re(u[c], eu);
        const int cr = j0 >> 3, ci = (nwp + j0) >> 3;  // chunks of K = j and K = nwp + j
        const uint32_t h = (j0 & 4) << 1;              // second half of the chunk: + 8 bytes
        oz_put4x2<NG>(Bs, bstr, oz_off<KP>(n, cr) + h, oz_off<KP>(nwp + n, ci) + h, 0u, v);
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = oz_im(u[c], eu);
        oz_put4x2<NG>(Bs, bstr, oz_off<KP>(nwp + n, cr) + h, oz_off<KP>(n, ci) + h, 0x80008000u, v);
      }
    }
    for (int t = 0; t < ntiles; ++t) {
      const int f0 = t * fpt, nfl = min(fpt, nFrot - f0), rows = nfl * nw;
      // ---- A1: rows (fl, m), K = [Re X[m][:] | Im X[m][:]]
      const bool xlow = xrow < rows && ((code_s[f0 + xfl] >> 30) & 1);
      if (xrow < rows) {
        int e = 1;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (xlow && 8 * xc8 + c == xm) xr[c].y = 0.0;  // a mirrored field's diagonal is real
          e = max(e, oz_cexp(xr[c]));
        }
        atomicMax(&xe_s[xrow], e);
        if (e >= Cfg::EMAX) fbad_s[xfl] = 1;
      }
      __syncthreads();
      if (xrow < 128) {
        const int ex = xe_s[xrow];
        long long v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = oz_re(xr[c], ex);
        oz_put8<NG>(As, ASTR, oz_off<KP>(xrow, xc8), v);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          v[c] = oz_im(xr[c], ex);
          if (xlow && 8 * xc8 + c > xm) v[c] = -v[c];
        }
        oz_put8<NG>(As, ASTR, oz_off<KP>(xrow, cpr + xc8), v);
      }
      fence_async_smem();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after();
        oz_issue<KP, NG>(tbase, smem_u32(As), smem_u32(Bs), ncol, ncol / 16, 0u);
        mma_commit(mb);
      }
      if (!wait_all(mb, phase, &abort_s, wait_ns)) break;
      phase ^= 1;
      tc_fence_after();
      // ---- T in fixed point: thread (field, m) holds columns c0.. of [Re T[m][:] | Im T[m][:]]; to its columns
      // through shared memory, [column][row]
      const bool live = 32 * quarter < rows;  // warp-uniform: some row of this warp is in use
      if (live) {
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          if (c < ncg) {
            long long q[4];
            oz_cols4<NG, KP>(tbase + lane_base + c0 + c, ncol, SH, q);
#pragma unroll
            for (int i = 0; i < 4; ++i) tq[(c0 + c + i) * OZ_LDQ + row] = q[i];
          }
        }
      }
      __syncthreads();
      // ---- A2: row (fl, n), K = m: [Re T[m][n] | -Im T[m][n]], thread as for X: 8 m of one row, both parts
      long long tr[8], ti[8];
      if (xrow < rows) {
        int te = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int m = 8 * xc8 + c, j = xfl * nw + m;
          tr[c] = m < nw ? tq[xm * OZ_LDQ + j] : 0;
          ti[c] = m < nw ? tq[(nwp + xm) * OZ_LDQ + j] : 0;
          const int ex = m < nw ? xe_s[j] : 0;
          te = max(te, max(oz_top(tr[c], ex), oz_top(ti[c], ex)));
        }
        atomicMax(&te_s[xrow], te);
      }
      __syncthreads();
      if (xrow < 128) {  // at the scale of the column of T: its rows' exponents come in, so that K has one exponent
        const int te = te_s[xrow];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int sh = xrow < rows && 8 * xc8 + c < nw ? 62 + xe_s[xfl * nw + 8 * xc8 + c] - te : 0;
          tr[c] = xrow < rows ? oz_shift(tr[c], sh) : 0;
          ti[c] = xrow < rows ? -oz_shift(ti[c], sh) : 0;
        }
        oz_put8<NG>(As, ASTR, oz_off<KP>(xrow, xc8), tr);
        oz_put8<NG>(As, ASTR, oz_off<KP>(xrow, cpr + xc8), ti);
      }
      tc_fence_before();
      fence_async_smem();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after();
        oz_issue<KP, NG>(tbase, smem_u32(As), smem_u32(Bs), ncol, ncol / 16, 0u);
        mma_commit(mb);
      }
      {  // the next tile's X while the products run
        const bool last = t + 1 == ntiles;
        const long long kn = last ? k + gridDim.x : k;
        if (kn < nk) {
          if (last && tid < (nw2 + 7) / 8) prefetch_l2(U + kn * strideU + tid * 8);
          load_x(kn, last ? 0 : t + 1);
        }
      }
      if (!wait_all(mb, phase, &abort_s, wait_ns)) break;
      phase ^= 1;
      tc_fence_after();
      // ---- D2: thread (fl, n) holds columns c0.. of [Re Y^H[n][:] | Im Y^H[n][:]]; staged, then written
      if (live) {
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          if (c < ncg) {
            long long s[4];
            oz_cols4<NG, KP>(tbase + lane_base + c0 + c, ncol, SH, s);
            const bool im = c0 + c >= nwp;
            long long* p = (im ? stim - nwp : stre) + row * ldst + c0 + c;
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = s[i];
          }
        }
      }
      tc_fence_before();
      __syncthreads();
#pragma unroll 2
      for (int e = tid; e < rows * nw; e += THR) {
        const int r = (int)__umulhi((uint32_t)e, magic), n = e - r * nw;  // row (field, m') and column n
        const int f = (int)__umulhi((uint32_t)r, magic), mr = r - f * nw;
        const int code = code_s[f0 + f], hmode = (code >> 28) & 3;
        const bool bad = code < 0 || fbad_s[f] || ubad_s;
        if (code >= 0 && hmode == 2 && n != mr) continue;
        int te = te_s[f * nw + n];
        const int o = (f * nw + n) * ldst + mr;  // Y[m'][n] = conj(Y^H[n][m'])
        long long re = stre[o], im = stim[o];
        if (hmode != 0) {  // + Y^H[m'][n] at the larger of the two scales, halved in the exponent
          const int p = r * ldst + n, d = te_s[r] - te, so = min(max(d, 0), 63), sp = min(max(-d, 0), 63);
          re = (re >> so) + (stre[p] >> sp);
          im = (im >> so) - (stim[p] >> sp);
          te = max(te, te_s[r]);
        }
        im = -im;
        const int E = 2 * EP - 62 + te + ue_s[n] + ue_s[mr] - 3 * Cfg::BIAS;
        Xbar[(k * ldf + f0 + f) * (long long)nw2 + mr * nw + n] =
            bad ? oz_nan(double2()) : oz_pack(double2(), re, im, hmode != 0 ? E - 1 : E);
      }
      __syncthreads();  // TMEM, the operands and the staging are free
      if (tid < 128) {
        xe_s[tid] = 1;
        te_s[tid] = 0;
      }
      if (tid < 32) {
        fbad_s[tid] = 0;
        if (t + 1 == ntiles) ue_s[tid] = 1;
      }
      if (tid == 0 && t + 1 == ntiles) ubad_s = 0;
      __syncthreads();
    }
  }
  if (abort_s) {  // a wait ran out: let the products already issued finish first
    if (tid == 0) mbar_wait(mb, phase, DRAIN_NS);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------
// 32 < nw <= 128: one field and one panel of PN = 32 columns at a time.
//   GEMM1  T = X U_P        A = [Re X | Im X] rows m       B = embedded U[:, P]
//   GEMM2  Y = U^dagger T   A = [Re U^T | Im U^T] rows m'  B = [[Re T, Im T], [Im T, -Re T]]
// K runs in stages of 16 complex rows ([16 Re | 16 Im]) through two operand buffers: while the tensor cores
// multiply one, all threads cut the next.  T stays in registers (fixed point) between the GEMMs, and the
// warps of TMEM lane quarter c write stages 2c and 2c + 1 of it as operand.  Rows >= nw of A are left as they
// are: they reach only accumulator rows that nothing reads.  Hermitian-part fields take the
// Hermitian part on input and write the lower triangle with its mirror, as rotate_panel does, so
// that the stored matrix is Hermitian bit for bit.
// ---------------------------------------------------------------------------------------
// Bound by the cutting.  One buffer of 32 rows, every product waited
// for: 17.3 ms at nw = 82 (double-float, 36 fields, 512 k-points) and 8.1 ms at nw = 48 (9 fields, 2 048);
// two buffers with all threads meeting at each stage: 17.7 and 7.0 ms; this, with a warp for the products and
// full / done barriers a stage, so that no cutting warp waits for another one: 14.0 and 5.7 ms (13.8 and 5.4 ms with one
// scale per matrix).
constexpr int OZ_PN = 32, OZ_WK = 512, OZ_THR = OZ_WK + 32;  // 16 warps at the operands, one for the products
template <int DF> constexpr int oz_large_smem() { return 2 * OzCfg<DF>::NG * (128 + 64) * 64 + 1024; }

// Largest exponents of the columns of U (mode 3) or of the rows of X as the kernel reads it: mode 0 as it is, 1 its
// Hermitian part (element (m, n) is part of row n, too), 2 the lower triangle and its mirror.  Coalesced, all 16 warps;
// a function of its own, so that its registers do not push the caller's out: nw = 82 as below 14.8 -> 14.1 ms.
template <int DF>
__device__ __noinline__ void oz_scales(const typename OzCfg<DF>::VI* __restrict__ M, int nw, int warp, int lane, int mode,
                                       int* e_s, int* bad_s) {
  typedef typename OzCfg<DF>::VI VI;
  int ec[4] = {1, 1, 1, 1}, er[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = warp + i * (OZ_WK / 32);
    er[i] = 1;
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // of a lower triangle only m >= n counts, of its diagonal the real part
      const int n = 32 * c + lane;
      if (m < nw && n < nw && (mode != 2 || m >= n)) {
        const VI v = M[m * nw + n];
        const int e = oz_cexp(mode == 2 && m == n ? oz_real(v) : v);
        er[i] = max(er[i], e);
        ec[c] = max(ec[c], e);
      }
    }
  }
  int top = 1;
  if (mode != 3)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = warp + i * (OZ_WK / 32);
      if (m >= nw) break;
      const int e = warp_max(er[i]);
      if (lane == 0) atomicMax(&e_s[m], e);
    }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (mode != 0 && 32 * c < nw) atomicMax(&e_s[32 * c + lane], ec[c]);
    top = max(top, ec[c]);
  }
  if (top >= OzCfg<DF>::EMAX) *bad_s = 1;
}

template <int DF>
__global__ void __launch_bounds__(OZ_THR, 1)
    rotate_oz_large(const typename OzCfg<DF>::VI* __restrict__ U, long long strideU,
                    const typename OzCfg<DF>::VI* __restrict__ X, int nFin, const int* __restrict__ fsel,
                    const int* __restrict__ herm, int nFrot, typename OzCfg<DF>::VO* __restrict__ Xbar, int nw, int nk,
                    long long per) {
  typedef OzCfg<DF> Cfg;
  typedef typename Cfg::VI VI;
  typedef typename Cfg::VO VO;
  typedef typename Cfg::PI PI;
  constexpr int NG = Cfg::NG, KP = 32;
  constexpr int SH = DF ? 6 : 14;  // K <= 256: |sum| <= 2^76 (FP64), 2^68 (double-float)
  constexpr int EP = SH + 112 - 8 * (NG - 1);
  constexpr uint32_t ASTR = 128 * 64, BSTR = 64 * 64, STAGE = NG * (ASTR + BSTR);  // A slices, then B slices
  constexpr int LDS = OZ_PN + 1;
  static_assert(2 * STAGE >= 2 * 128 * LDS * 8, "the staging overlays the operand buffers");
  extern __shared__ __align__(1024) unsigned char smo[];
  unsigned char* As = smo + ((1024u - (smem_u32(smo) & 1023u)) & 1023u);
  long long* stre = reinterpret_cast<long long*>(As);  // staging: [m'][n] re plane, then im plane
  long long* stim = stre + 128 * LDS;
  __shared__ __align__(8) uint64_t mbar[4];  // full[2]: an arrival a warp; done[2]: the products' commit
  __shared__ uint32_t tmem_base_s;
  // largest exponents of each column of U, each row of X and each column of the panel of T (0: zero); non-finite
  // elements of U and of the field
  __shared__ int ue_s[128], xe_s[128], te_s[OZ_PN];
  __shared__ int abort_s, ubad_s, fbad_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full = smem_u32(mbar), done = full + 16;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full + 8 * i), "r"(OZ_WK / 32) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(done + 8 * i) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_s = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  const int nw2 = nw * nw, np = (nw + OZ_PN - 1) / OZ_PN, nst = (nw + 15) / 16;
  const int quarter = warp & 3, half = warp >> 3, sub = (warp >> 2) & 1;  // columns 32 half + 16 sub ..
  const uint32_t lane_base = ((uint32_t)(32 * quarter) << 16) + 32 * half + 16 * sub;
  const int row = 32 * quarter + lane;
  const unsigned long long wait_ns = g_tc_wait_ns;
  volatile int* ab = &abort_s;
  uint32_t g = 0;  // stages so far: stage g in buffer g & 1, phase g >> 1 of its barriers
  long long kprev = -1, fprev = -1;
  const long long total = (long long)nk * nFrot * np;
  const long long u1 = min(total, (blockIdx.x + 1) * per);
  // task of the A operand: 8 columns of one part (0 re, 1 im) of one row (8 lanes take 8 rows); of the embedded
  // U panel: rows bj, bj + 1 of one part of column n0 + lane
  const int am = (tid >> 5) * 8 + (tid & 7), akc = (tid >> 3) & 3, apart = akc >> 1, aj = 8 * (akc & 1);
  const int bj = 2 * (warp & 7), bpart = warp >> 3;
  PI xr[8], br[2];
  // A wait that runs out sets abort_s: the warps then skip operands and accumulators, but meet at every barrier
  // until the next unit, where all leave together.
  bool ok = true;
  auto wait_stage = [&](uint32_t x) {  // all products of stage x are done (x < g)
    if (lane == 0) ok = ok && kt_wait(done + 8 * (x & 1), (x >> 1) & 1u, ab, wait_ns);
    ok = __shfl_sync(0xffffffffu, ok, 0);
  };
  auto stage_full = [&]() {  // this warp's part of the stage is written
    fence_async_smem();
    tc_fence_before();
    __syncwarp();
    if (lane == 0 && ok) mbar_arrive(full + 8 * (g & 1));
    ++g;
  };
  auto wsync = [&]() { named_sync(1, OZ_WK); };
  if (warp == OZ_WK / 32) {
    // ---- products: two GEMMs of nst stages a unit
    if (lane == 0) {
      const long long nu = u1 - blockIdx.x * per;
      for (long long u = 0; u < 2 * nu && ok; ++u)
        for (int i = 0; i < nst; ++i, ++g) {
          ok = kt_wait(full + 8 * (g & 1), (g >> 1) & 1u, ab, wait_ns);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = smem_u32(As + (g & 1) * STAGE);
          oz_issue_all<KP, NG, 64>(tbase, st, st + NG * ASTR, (uint32_t)(i > 0));
          mma_commit(done + 8 * (g & 1));
        }
      if (g > 0) mbar_wait(done + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1u, DRAIN_NS);  // no product in flight at exit
    }
    __syncwarp();
  } else {
  for (long long u = blockIdx.x * per; u < u1; ++u) {
    const int P = (int)(u % np), f = (int)((u / np) % nFrot);
    const long long k = u / ((long long)np * nFrot);
    const int fs = fsel[f], hm = herm[f];
    const bool fok = fs >= 0 && fs < nFin;  // selection lives in device memory: validate here
    const int inmode = (hm & 4) ? 2 : ((hm & 3) != 0 ? 1 : 0);
    const VI* Xf = X + (k * nFin + (fok ? fs : 0)) * (long long)nw2;
    const VI* Uk = U + k * strideU;
    const int n0 = P * OZ_PN;
    // ---- largest exponents of U_k and of the field (kept while the CTA stays on them)
    const bool newk = k != kprev, newf = newk || f != fprev;
    if (named_any(1, OZ_WK, !ok || *ab)) break;
    if (tid < 128) {
      if (newk) ue_s[tid] = 1;
      if (newf) xe_s[tid] = 1;
    }
    if (tid < OZ_PN) te_s[tid] = 0;
    if (tid == 0) {
      if (newk) ubad_s = 0;
      if (newf) fbad_s = 0;
    }
    wsync();
    if (newk) oz_scales<DF>(Uk, nw, warp, lane, 3, ue_s, &ubad_s);
    if (newf) oz_scales<DF>(Xf, nw, warp, lane, inmode, xe_s, &fbad_s);
    kprev = k;
    fprev = f;
    const PI* Xp = reinterpret_cast<const PI*>(Xf) + apart;
    const PI* Up = reinterpret_cast<const PI*>(Uk);
    const PI* Xa = Xp + 2 * (am * nw + aj);
    auto load_x = [&](int i) {  // stage i of GEMM1: X and the rows of U[:, P]
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int j = 16 * i + aj + q;
        xr[q] = oz_zero(PI());
        if (am < nw && j < nw) xr[q] = inmode == 2 && j > am ? Xp[2 * (j * nw + am)] : Xa[2 * (16 * i + q)];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = 16 * i + bj + q;
        br[q] = n0 + lane < nw && j < nw ? Up[2 * (j * nw + n0 + lane) + bpart] : oz_zero(PI());
      }
    };
    int eua = 0;  // exponent of the column of U that this thread's row of U^H is
    auto load_uh = [&](int i) {  // stage i of GEMM2: row m' of U^H: U[j][m']
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int j = 16 * i + aj + q;
        xr[q] = am < nw && j < nw ? Up[2 * (j * nw + am) + apart] : oz_zero(PI());
      }
    };
    auto put_uh = [&]() {
      if (am < nw && ok) {
        long long v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = oz_part(xr[q], eua);
        oz_put8<NG>(As + (g & 1) * STAGE, ASTR, oz_off<KP>(am, akc), v);
      }
    };
    load_x(0);
    wsync();
    const int ex = xe_s[am], eub = ue_s[n0 + lane];
    eua = ue_s[am];
    // ---- GEMM1
    for (int i = 0; i < nst; ++i) {
      if (i >= 2) wait_stage(g - 2);  // (the previous unit's stages are done)
      unsigned char* A = As + (g & 1) * STAGE;
      unsigned char* B = A + NG * ASTR;
      if (am < nw && ok) {
        long long v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = oz_part(xr[q], ex);
        if (inmode == 2 && apart) {  // the mirror's conjugate, the real diagonal
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int j = 16 * i + aj + q;
            v[q] = j > am ? -v[q] : j == am ? 0 : v[q];
          }
        }
        if (inmode == 1) {  // Hermitian part of the input
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int j = 16 * i + aj + q;
            if (j < nw) {
              const long long o = oz_part(Xp[2 * (j * nw + am)], ex);
              v[q] = (apart ? v[q] - o : v[q] + o) >> 1;
            }
          }
        }
        oz_put8<NG>(A, ASTR, oz_off<KP>(am, akc), v);
      }
      if (ok) {  // embedded U[:, P]: Re at (n, re K) and (32 + n, im K), Im at (32 + n, re K) and, negated, at (n, im K)
        const int rc = bj >> 3;
        const uint32_t h = (bj & 7) * 2;
        oz_put2x2<NG>(B, BSTR, oz_off<KP>(bpart ? 32 + lane : lane, rc) + h,
                      oz_off<KP>(bpart ? lane : 32 + lane, 2 + rc) + h, bpart ? 0x80008000u : 0u, oz_part(br[0], eub),
                      oz_part(br[1], eub));
      }
      stage_full();
      if (i + 1 < nst) load_x(i + 1);
      else load_uh(0);
    }
    // the first stage of U^H while the last products run
    wait_stage(g - 2);
    put_uh();
    load_uh(1);
    wait_stage(g - 1);
    tc_fence_after();
    // ---- T: thread (row j) holds 16 columns n of Re (half 0) or Im (half 1) T[j][n0 + 16 sub ..]
    long long q[16];
    const bool live = 32 * quarter < nw;
    const int exr = xe_s[row];
    if (live && ok) {
      int top = 0;
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        oz_cols4<NG, 256>(tbase + lane_base + c, 64, SH, q + c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (row >= nw) q[c + i] = 0;
          const int e = warp_max(oz_top(q[c + i], exr));
          if (lane == c + i) top = e;
        }
      }
      if (lane < 16) atomicMax(&te_s[16 * sub + lane], top);
    }
    wsync();
    // to the scale of the column of T: its row's exponent comes in, so that K has one exponent
    if (live)
#pragma unroll
      for (int c = 0; c < 16; ++c) q[c] = oz_shift(q[c], 62 + exr - te_s[16 * sub + c]);
    // lanes l and l + 16 exchange half of their columns, so that the 16 rows of a stage lie on all lanes: lane l
    // then holds columns 16 sub + 8 (l >> 4) .. + 7 of rows l & 15 (q[0 .. 7]) and 16 + (l & 15) (q[8 .. 15])
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const long long o = __shfl_xor_sync(0xffffffffu, lane < 16 ? q[8 + i] : q[i], 16);
      if (lane < 16) q[8 + i] = o;
      else q[i] = o;
    }
    // ---- GEMM2
    const int jl = lane & 15;
    const int ka = half * 16 + jl, kb = (1 - half) * 16 + jl;  // K of the n and of the 32 + n rows
    const uint32_t flip = half ? 0u : 0x80008000u;             // -Re T at (32 + n, im K)
    const bool odd = lane & 1;  // even lanes write column n of rows j, j + 1, odd lanes column n + 1 of j - 1, j
    for (int i = 0; i < nst; ++i) {
      if (i > 0) {
        if (i >= 2) wait_stage(g - 2);
        put_uh();
        if (i + 1 < nst) load_uh(i + 1);
      }
      if (quarter == i >> 1 && ok) {  // this quarter's rows j
        unsigned char* B = As + (g & 1) * STAGE + NG * ASTR;
        unsigned char* b0 = B + (ka & 6) * 2;
        unsigned char* b1 = B + (kb & 6) * 2;
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
          const long long a = i & 1 ? q[8 + c] : q[c], b = i & 1 ? q[9 + c] : q[c + 1];
          const long long o = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
          const unsigned long long wa = oz_bias(odd ? o : a), wb = oz_bias(odd ? b : o);
          const int n = 16 * sub + 8 * (lane >> 4) + c + odd;
          unsigned char* p0 = b0 + oz_off<KP>(n, ka >> 3);
          unsigned char* p1 = b1 + oz_off<KP>(32 + n, kb >> 3);
#pragma unroll
          for (int s = 0; s < NG; ++s) {
            const uint32_t d = oz_dig2(oz_word(wa, s), oz_word(wb, s), 3 - (s & 3));
            *reinterpret_cast<uint32_t*>(p0 + s * BSTR) = d;
            *reinterpret_cast<uint32_t*>(p1 + s * BSTR) = d ^ flip;
          }
        }
      }
      stage_full();
    }
    wait_stage(g - 2);
    wait_stage(g - 1);
    tc_fence_after();
    // ---- Y: thread (row m') holds 16 columns of Re or Im of Y[m'][n0 ..]; staged, then written by rows
    if (live && ok) {
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        long long s[4];
        oz_cols4<NG, 256>(tbase + lane_base + c, 64, SH, s);
        long long* p = (half ? stim : stre) + row * LDS + 16 * sub + c;
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = s[i];
      }
    }
    tc_fence_before();
    wsync();
    const bool bad = !fok || fbad_s || ubad_s;
    auto yexp = [&](int nl) { return 2 * EP - 62 + te_s[nl] + ue_s[n0 + nl] - 3 * Cfg::BIAS; };  // less that of row m'
    VO* dst = Xbar + (k * nFrot + f) * (long long)nw2;
    const int mode = hm & 3, n = n0 + lane, E = yexp(lane);
    for (int m = warp; m < nw && ok; m += OZ_WK / 32) {
      if (n >= nw || (mode != 0 && n > m) || (mode == 2 && n != m)) continue;
      VO y = oz_pack(VO(), stre[m * LDS + lane], stim[m * LDS + lane], E + ue_s[m]);
      if (mode != 0 && m == n) y.y = 0;
      dst[m * nw + n] = bad ? oz_nan(y) : y;
    }
    if (mode == 1 && ok) {  // the mirror: row n of the panel, columns m > n
      for (int nl = warp; nl < OZ_PN && n0 + nl < nw; nl += OZ_WK / 32) {
        const int En = yexp(nl);
        for (int m = n0 + nl + 1 + lane; m < nw; m += 32) {
          const VO y = oz_pack(VO(), stre[m * LDS + nl], -stim[m * LDS + nl], En + ue_s[m]);
          dst[(n0 + nl) * nw + m] = bad ? oz_nan(y) : y;
        }
      }
    }
  }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(512) : "memory");
  }
}
