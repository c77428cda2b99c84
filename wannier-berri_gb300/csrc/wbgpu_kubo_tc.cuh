#pragma once
// Kubo band sums on the tensor cores (mixed path; calculators/dynamic.py:97-98,
//   restot += factor_omega @ (factor_Efermi x M)):
//   out[w][j] += sum_r F[w][r] G[r][j] per k-point,  F = f_w(dE_r), G[r][(e, c)] = f_E[r][e] M[r][c]
// over the pair records of wbgpu_kubo.cu (dE FP64, f_E and M FP32).  Real embedding with two K
// entries per record (Re F, Im F):
//   A[w][2r + p]      = p ? Im F : Re F                                  M = 128 frequencies
//   B[2j + q][2r + p] = [[Re G, -Im G], [Im G, Re G]][q][p]              N = 2 x (<= 104 columns j)
//   D[w][2j + q]      = q ? Im (F G)[w][j] : Re (F G)[w][j]
// F is formed in FP32 from dE - w taken as (dE_hi - w_hi) + (dE_lo - w_lo) (double-float halves:
// the difference to FP32 accuracy without the FP64 pipe).  Operands are split into TF32 hi + lo
// (3xTF32) as in the rotation.  The records of one k-point run in fills of KT_RC = 16 (K = 32, four
// MMA K-steps, three products each) to a fresh TMEM accumulator each, so no accumulator takes more
// than twelve truncating steps (at most ~3e-7 relative drift toward zero).  The epilogue adds each
// fill with round-to-nearest into per-k-point FP32 sums, and adds those to the fixed-point output
// once per k-point (order-independent: the same bits in any grid shape).
// Roles (one CTA of six warpgroups per SM): warps 0-7 epilogue (TMEM lane quarter = warp & 3, column
// half = warp >> 2), which keep their 104 sums a thread in registers (setmaxnreg: 144 a thread; through
// shared memory the sums would take 1 664 of a fill's cycles and the space of the second operand
// stage); warps 8-19 operand producers, one barrier among them per fill, records copied three fills
// ahead; one thread of the last warpgroup issues the MMAs of a fill as soon as its stage is full and
// its accumulator drained.  Two stages and two accumulators alternate: a fill is formed while the
// previous one multiplies and the one before that is drained.  Every mbarrier wait is bounded by the
// kernel's wait limit, as in the rotation.
// Bound by the producers' instruction streams (one 4^3 block: issue slots 50% active, tensor pipe 30%).  At 400
// frequencies x 11 levels x 9 components, num_wann 96 and 512 k-points: 27.8 ms with eight-record
// chunks, three producer barriers each and the sums in shared memory; 11.9 ms with fills formed in one
// go and the sums in registers by eight producer warps, 10.7 ms by these twelve.
constexpr int KT_M = 128, KT_CT = 104, KT_NMAX = 2 * KT_CT, KT_RC = 16, KT_K = 2 * KT_RC, KT_NST = 2;
constexpr int KT_LBO = 128;                          // K-adjacent core matrices contiguous
constexpr int KT_SBO = (KT_K / 4) * KT_LBO + 16;     // 8-row groups, 16 bytes apart in banks
constexpr int KT_A_BYTES = (KT_M / 8) * KT_SBO;      // one copy (hi or lo) of F
constexpr int KT_B_BYTES = (KT_NMAX / 8) * KT_SBO;   // one copy of the embedded G
constexpr int KT_STAGE = 2 * KT_A_BYTES + 2 * KT_B_BYTES;
// a fill's records, copied ahead: dE, f_E of the tile's levels (<= KT_EMAX), M (<= KT_NCMAX)
constexpr int KT_EMAX = 16, KT_NCMAX = 27;
constexpr int KT_REC_FE = KT_RC * 8, KT_REC_M = KT_REC_FE + KT_RC * KT_EMAX * 4;
constexpr int KT_REC_BYTES = KT_REC_M + KT_RC * KT_NCMAX * 8;
constexpr int KT_NREC = 4;  // record buffers: copies run KT_NREC - 1 fills ahead (cp_async_wait_ahead)
// a warp's way from registers to the output: 32 rows of 16 columns, rows 80 bytes apart (16-byte
// accesses of eight rows fall on distinct banks)
constexpr int KT_FLUSH_LD = 20, KT_FLUSH_BYTES = 32 * KT_FLUSH_LD * 4;
constexpr int KT_EPI = 256, KT_PROD0 = KT_EPI, KT_PRODN = 384, KT_MMA0 = KT_PROD0 + KT_PRODN, KT_THR = KT_MMA0 + 128;
constexpr int KT_SMEM = KT_NST * KT_STAGE + KT_NREC * KT_REC_BYTES + (KT_EPI / 32) * KT_FLUSH_BYTES;
constexpr uint32_t KT_TMEM_COLS = 512;               // accumulator of fill t at column 256 (t & 1)
// registers a thread at launch, and after the roles have split them: the shares fit the launch's total
constexpr int KT_REG_LAUNCH = 80, KT_REG_EPI = 144, KT_REG_PROD = 56, KT_REG_MMA = 24;
static_assert(KT_EPI * KT_REG_EPI + KT_PRODN * KT_REG_PROD + 128 * KT_REG_MMA <= KT_THR * KT_REG_LAUNCH,
              "register shares beyond the launch's would wait forever");
static_assert(KT_SMEM <= 220 * 1024, "operand stages, records and the flush buffers must fit one CTA's shared memory");
static_assert(KT_STAGE % 16 == 0 && KT_REC_BYTES % 16 == 0 && KT_REC_FE % 16 == 0 && KT_REC_M % 16 == 0, "alignment");
static_assert(KT_RC * KT_EMAX <= KT_PRODN, "at most one f_E value a producer thread");
static_assert(KT_PRODN % KT_M == 0, "one frequency row a producer thread");
constexpr int KT_BPT = (KT_CT * (KT_RC / 2) + KT_PRODN - 1) / KT_PRODN;  // pieces of G a producer thread

WBG_D uint64_t kt_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(KT_LBO >> 4) << 16) | ((uint64_t)(KT_SBO >> 4) << 32) |
         (1ull << 46);
}
WBG_D uint32_t kt_off(int r, int k) {  // byte offset of element (row r, K index k % 4 == 0) of an operand
  return (uint32_t)((r >> 3) * KT_SBO + (k >> 2) * KT_LBO + (r & 7) * 16);
}
WBG_D void kt_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
WBG_D void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
WBG_D void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
WBG_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// every group but the newest KT_NREC - 2 complete (KT_NREC = 4): the next fill's records
WBG_D void cp_async_wait_ahead() { asm volatile("cp.async.wait_group 2;" ::: "memory"); }

// Records r0 .. r0 + rn - 1 of a k-point into a record buffer: dE, f_E of levels e0 .. e0 + ne - 1, the
// NC components of M (record by record, as they lie); thread i of KT_PRODN.
WBG_D void kt_stage_records(unsigned char* rb, const double* rec_dE, const float* rec_fE, const float2* rec_M,
                            long long rbase, int rn, int nEF, int e0, int ne, int NC, int i) {
  if (i < rn) cp_async8(rb + 8 * i, rec_dE + rbase + i);
  const int r = i / KT_EMAX, e = i % KT_EMAX;
  if (r < rn && e < ne) cp_async4(rb + KT_REC_FE + 4 * i, rec_fE + (rbase + r) * nEF + e0 + e);
  for (int p = i; p < rn * NC; p += KT_PRODN) cp_async8(rb + KT_REC_M + 8 * p, rec_M + rbase * NC + p);
}

// Bounded wait of the Kubo kernel: mbarrier.try_wait with a suspend-time hint, so that a waiting
// thread sleeps in the barrier unit (up to 20 us per try) instead of spinning; gives up on an abort
// by another role or after limit_ns, recording the timeout like pipe_wait.
WBG_D bool kt_wait(uint32_t mb, uint32_t parity, volatile int* abort_s, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mb), "r"(parity), "r"(20000u)
        : "memory");
    if (ok) return true;
    if (*abort_s) return false;
    if (global_ns() - t0 > limit_ns) {
      *abort_s = 1;
      atomicOr(&g_wbg_device_flags, (unsigned)WBG_DEVICE_FLAG_TC_TIMEOUT);
      return false;
    }
  }
}

// x rounded to TF32 (10-bit mantissa, to nearest, ties away from zero: the result of cvt.rna.tf32.f32
// for finite x) with two integer operations on the full-rate integer pipe
WBG_D uint32_t tf32_rna_int(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
// four K-consecutive values split as hi + lo (both TF32) into the two operand copies, as put_split4
WBG_D void kt_split4(unsigned char* hi, unsigned char* lo, uint32_t off, float a, float b, float c, float d) {
  uint4 h, l;
  h.x = tf32_rna_int(a);
  h.y = tf32_rna_int(b);
  h.z = tf32_rna_int(c);
  h.w = tf32_rna_int(d);
  l.x = tf32_rna_int(a - __uint_as_float(h.x));
  l.y = tf32_rna_int(b - __uint_as_float(h.y));
  l.z = tf32_rna_int(c - __uint_as_float(h.z));
  l.w = tf32_rna_int(d - __uint_as_float(h.w));
  *reinterpret_cast<uint4*>(hi + off) = h;
  *reinterpret_cast<uint4*>(lo + off) = l;
}

// the operand rows (Re g0, -Im g0, Re g1, -Im g1) and (Im g0, Re g0, Im g1, Re g1): four splits (rounding to
// nearest is symmetric, so the split of -x is the negated split of x)
WBG_D void kt_split_G(unsigned char* hi, unsigned char* lo, uint32_t off, float2 g0, float2 g1) {
  uint4 h, l;
  h.x = tf32_rna_int(g0.y);
  h.y = tf32_rna_int(g0.x);
  h.z = tf32_rna_int(g1.y);
  h.w = tf32_rna_int(g1.x);
  l.x = tf32_rna_int(g0.y - __uint_as_float(h.x));
  l.y = tf32_rna_int(g0.x - __uint_as_float(h.y));
  l.z = tf32_rna_int(g1.y - __uint_as_float(h.z));
  l.w = tf32_rna_int(g1.x - __uint_as_float(h.w));
  *reinterpret_cast<uint4*>(hi + off + 16) = h;
  *reinterpret_cast<uint4*>(lo + off + 16) = l;
  *reinterpret_cast<uint4*>(hi + off) = make_uint4(h.y, h.x ^ 0x80000000u, h.w, h.z ^ 0x80000000u);
  *reinterpret_cast<uint4*>(lo + off) = make_uint4(l.y, l.x ^ 0x80000000u, l.w, l.z ^ 0x80000000u);
}

WBG_D void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
WBG_D void tmem_ld_wait8(uint32_t* r) {
  asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
               "+r"(r[7])::"memory");
}

template <int N>
WBG_D void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
WBG_D void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// f_w of one record for frequency w: dE - w and -dE - w from the double-float halves; formula
// WBG_DYN_OPTCOND dE / (dE - w - i eta), WBG_DYN_SHC_SIMPLE (every spin Hall kind)
// 1 / (-dE - w - i eta) / 2, WBG_DYN_SHIFT smear(-dE - w) + smear(dE - w), otherwise
// smear(-dE - w); Lorentzian or Gaussian (the frequency factors of wbgpu_kubo.cu in FP32)
// The products are rounded by name: fused into the sums and splits that take them they would give other bits.
template <int FORMULA, bool GAUSS>
WBG_D float2 kt_factor(float deh, float del, float wh, float wl, float eta) {
  const float dp = (deh - wh) + (del - wl), dm = (-deh - wh) + (-del - wl);
  if (FORMULA == WBG_DYN_OPTCOND || FORMULA == WBG_DYN_SHC_SIMPLE) {
    const float d = FORMULA == WBG_DYN_OPTCOND ? dp : dm;
    const float den = __fdividef(1.0f, fmaf(d, d, __fmul_rn(eta, eta)));
    const float cre = __fmul_rn(d, den);
    float cim = __fmul_rn(eta, den);
    if (GAUSS) {
      const float x = d / eta;
      cim = fabsf(d) < eta * 14.142135623730951f ? __fmul_rn(1.7724538509055160f / eta, __expf(-__fmul_rn(x, x))) : 0.0f;
    }
    const float s = FORMULA == WBG_DYN_OPTCOND ? deh + del : 0.5f;
    return make_float2(__fmul_rn(s, cre), __fmul_rn(s, cim));
  }
  auto sm = [&](float x) {
    if (GAUSS) {
      const float y = x / eta;
      return fabsf(x) < eta * 14.142135623730951f ? __fmul_rn(0.5641895835477563f / eta, __expf(-__fmul_rn(y, y))) : 0.0f;
    }
    return __fmul_rn(__fmul_rn(0.3183098861837907f, eta), __fdividef(1.0f, fmaf(x, x, __fmul_rn(eta, eta))));
  };
  float v = sm(dm);
  if (FORMULA == WBG_DYN_SHIFT) v += sm(dp);
  return make_float2(v, 0.0f);
}

// A: one frequency row of F, records (2q, 2q + 1) -> K entries 4q .. 4q + 3 for q = q0, q0 + KT_PRODN / KT_M ..
template <int FORMULA, bool GAUSS>
WBG_D void kt_form_A(unsigned char* Ah, unsigned char* Al, const float2* de, int row, int q0, int rn, float wh, float wl,
                     float eta) {
#pragma unroll
  for (int i = 0; i < (KT_RC / 2 * KT_M + KT_PRODN - 1) / KT_PRODN; ++i) {
    const int q = q0 + i * (KT_PRODN / KT_M);
    if (2 * q >= (rn + 7) / 8 * 8) break;  // K-steps that are not issued
    const float4 d = reinterpret_cast<const float4*>(de)[q];
    float2 f0 = make_float2(0.f, 0.f), f1 = make_float2(0.f, 0.f);
    if (2 * q < rn) f0 = kt_factor<FORMULA, GAUSS>(d.x, d.y, wh, wl, eta);
    if (2 * q + 1 < rn) f1 = kt_factor<FORMULA, GAUSS>(d.z, d.w, wh, wl, eta);
    kt_split4(Ah, Al, kt_off(row, 4 * q), f0.x, f0.y, f1.x, f1.y);
  }
}

__global__ void __launch_bounds__(KT_THR, 1)
    kubo_tc(const double* __restrict__ rec_dE, const float* __restrict__ rec_fE, const float2* __restrict__ rec_M,
            const int* __restrict__ count, int P, int nk, int kchunk, const double* __restrict__ omega, int nOmega,
            int nEF, int NC, int ctile, float eta, int gaussian, int fgroup, wbg_u64* __restrict__ out) {
  extern __shared__ __align__(128) unsigned char smk[];
  __shared__ __align__(8) uint64_t bar_s[2 * KT_NST + 4];  // full[KT_NST] empty[KT_NST] accfull[2] accfree[2]
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int w0 = blockIdx.x * KT_M, col0 = blockIdx.z * ctile;
  const int ncol = nEF * NC, nct = min(ctile, ncol - col0);  // ctile <= KT_CT
  const int N = (2 * nct + 15) / 16 * 16;
  const long long k0 = (long long)blockIdx.y * kchunk, k1 = min((long long)nk, k0 + kchunk);
  auto bar = [&](int i) { return smem_u32(&bar_s[i]); };
  enum { FULL = 0, EMPTY = KT_NST, ACCFULL = 2 * KT_NST, ACCFREE = 2 * KT_NST + 2 };
  if (tid == 0) {
    for (int i = 0; i < KT_NST; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(FULL + i)), "r"(KT_PRODN / 32) : "memory");
    for (int i = 0; i < KT_NST; ++i) mbar_init(bar(EMPTY + i));  // one arrival: the MMA commit
    for (int i = 0; i < 2; ++i) mbar_init(bar(ACCFULL + i));
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(ACCFREE + i)), "r"(KT_EPI / 32) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_s = 0;
  }
  for (int i = tid; i < KT_SMEM / 16; i += KT_THR)  // padding rows and columns stay zero
    reinterpret_cast<uint4*>(smk)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (warp == KT_MMA0 / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(KT_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  const unsigned long long wait_ns = g_tc_wait_ns;
  volatile int* ab = &abort_s;
  if (warp >= KT_MMA0 / 32) {
    // ================= MMA issue =================
    setmaxnreg_dec<KT_REG_MMA>();
    if (tid == KT_MMA0) {
      const uint32_t idesc =
          (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(KT_M >> 4) << 24);
      int t = 0;  // fill sequence number: stage and accumulator t & 1
      bool ok = true;
      for (long long k = k0; k < k1 && ok; ++k) {
        const int nrec = count[k];
        for (int r0 = 0; r0 < nrec; r0 += KT_RC, ++t) {
          const int s = t & 1;
          const uint32_t par = (uint32_t)((t >> 1) & 1);
          ok = kt_wait(bar(FULL + s), par, ab, wait_ns) &&
               (t < 2 || kt_wait(bar(ACCFREE + s), par ^ 1u, ab, wait_ns));
          if (!ok) break;
          tc_fence_after();
          const uint32_t ah = smem_u32(smk + s * KT_STAGE), al = ah + KT_A_BYTES, bh = al + KT_A_BYTES,
                         bl = bh + KT_B_BYTES;
          const uint32_t D = tbase + (uint32_t)(256 * s);
          const int ks = (min(KT_RC, nrec - r0) + 7) / 8 * 2;  // K-steps of 8 with records
          for (int i = 0; i < ks; ++i) {
            const uint32_t so = (uint32_t)i * 2 * KT_LBO;
            kt_mma(D, kt_desc(ah + so), kt_desc(bh + so), idesc, i > 0);
            kt_mma(D, kt_desc(al + so), kt_desc(bh + so), idesc, 1);
            kt_mma(D, kt_desc(ah + so), kt_desc(bl + so), idesc, 1);
          }
          mma_commit(bar(EMPTY + s));
          mma_commit(bar(ACCFULL + s));
        }
      }
      // no product in flight at exit: the last fill's commit
      if (t > 0) mbar_wait(bar(EMPTY + ((t - 1) & 1)), (uint32_t)(((t - 1) >> 1) & 1), DRAIN_NS);
    }
    __syncwarp();
  } else if (warp >= KT_PROD0 / 32) {
    // ================= operand producers =================
    setmaxnreg_dec<KT_REG_PROD>();
    const int pt = tid - KT_PROD0;
    const int prow = pt % KT_M, q0 = pt / KT_M;  // row of F; its first pair of records
    const bool arow = w0 + prow < nOmega;
    const double om = arow ? omega[w0 + prow] : 0.0;
    const float wh = (float)om, wl = (float)(om - (double)wh);
    const int e0 = col0 / NC, ne = (col0 + nct - 1) / NC - e0 + 1;  // the tile's levels (<= KT_EMAX)
    // this thread's pieces of G: column j of the tile, records (2q, 2q + 1): the offsets of the operand
    // rows 2j and 2j + 1, of f_E and of M in their buffers (bytes; -1: none)
    int boff[KT_BPT], foff[KT_BPT], moff[KT_BPT];
#pragma unroll
    for (int i = 0; i < KT_BPT; ++i) {
      const int idx = pt + i * KT_PRODN, q = idx / nct, j = idx - q * nct;
      const int e = (col0 + j) / NC, c = col0 + j - e * NC;
      boff[i] = q < KT_RC / 2 ? (int)kt_off(2 * j, 4 * q) : -1;
      foff[i] = (2 * q * KT_EMAX + e - e0) * 4;
      moff[i] = (2 * q * NC + c) * 8;
    }
    // the fill sequence: (k-point, first record) over the CTA's k-points with records
    auto skip_empty = [&](long long& kk, int& rr, int& cc) {  // cc: count[kk]
      while (rr >= cc && ++kk < k1) {
        rr = 0;
        cc = count[kk];
      }
    };
    auto rbuf = [&](int tt) { return smk + KT_NST * KT_STAGE + (tt % KT_NREC) * KT_REC_BYTES; };
    long long kc = k0, kf;  // the fill being formed, and the next one to copy
    int rc = 0, cc = k0 < k1 ? count[k0] : 0, rf, cf;
    skip_empty(kc, rc, cc);
    kf = kc;
    rf = rc;
    cf = cc;
    auto prefetch = [&](int tt) {  // the records of fill kf / rf into buffer tt, then advance kf / rf
      if (kf < k1) {
        kt_stage_records(rbuf(tt), rec_dE, rec_fE, rec_M, kf * (long long)P + rf, min(KT_RC, cf - rf), nEF, e0, ne, NC,
                         pt);
        rf += KT_RC;
        skip_empty(kf, rf, cf);
      }
      cp_async_commit();  // one group per fill, empty past the last
    };
    // dE of buffer tt into (hi, lo) in place, by the threads that copied them
    auto split_dE = [&](int tt) {
      if (pt < KT_RC) {
        const double de = reinterpret_cast<const double*>(rbuf(tt))[pt];
        const float h = (float)de;
        reinterpret_cast<float2*>(rbuf(tt))[pt] = make_float2(h, (float)(de - (double)h));
      }
    };
    for (int tt = 0; tt < KT_NREC - 1; ++tt) prefetch(tt);
    cp_async_wait_ahead();
    split_dE(0);
    named_sync(1, KT_PRODN);
    for (int t = 0; kc < k1; ++t) {
      const int s = t & 1, rn = min(KT_RC, cc - rc);
      bool ok = true;
      if (lane == 0 && t >= KT_NST) ok = kt_wait(bar(EMPTY + s), (uint32_t)(((t >> 1) - 1) & 1), ab, wait_ns);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      prefetch(t + KT_NREC - 1);  // its buffer held fill t - 1, read before the last barrier
      if (ok) {
        unsigned char* Ah = smk + s * KT_STAGE;
        unsigned char* Al = Ah + KT_A_BYTES;
        unsigned char* Bh = Al + KT_A_BYTES;
        unsigned char* Bl = Bh + KT_B_BYTES;
        const unsigned char* rb = rbuf(t);
        const float2* de = reinterpret_cast<const float2*>(rb);
        if (arow) {
#define WBG_KT_A(F)                                                                       \
  do {                                                                                    \
    if (gaussian) kt_form_A<F, true>(Ah, Al, de, prow, q0, rn, wh, wl, eta);              \
    else kt_form_A<F, false>(Ah, Al, de, prow, q0, rn, wh, wl, eta);                      \
  } while (0)
          if (fgroup == WBG_DYN_OPTCOND) WBG_KT_A(WBG_DYN_OPTCOND);
          else if (fgroup == WBG_DYN_SHC_SIMPLE) WBG_KT_A(WBG_DYN_SHC_SIMPLE);
          else if (fgroup == WBG_DYN_SHIFT) WBG_KT_A(WBG_DYN_SHIFT);
          else WBG_KT_A(WBG_DYN_INJECTION);
#undef WBG_KT_A
        }
        // B: rows 2j, 2j + 1 for column j of the tile, records (2q, 2q + 1)
#pragma unroll
        for (int i = 0; i < KT_BPT; ++i) {
          if (boff[i] < 0) continue;
          const int r = foff[i] / (KT_EMAX * 4);  // = 2q
          if (r >= (rn + 7) / 8 * 8) continue;    // K-steps that are not issued
          const float fe0 = *reinterpret_cast<const float*>(rb + KT_REC_FE + foff[i]);
          const float fe1 = *reinterpret_cast<const float*>(rb + KT_REC_FE + foff[i] + KT_EMAX * 4);
          const float2 m0 = *reinterpret_cast<const float2*>(rb + KT_REC_M + moff[i]);
          const float2 m1 = *reinterpret_cast<const float2*>(rb + KT_REC_M + moff[i] + 8 * NC);
          float2 g0 = make_float2(0.f, 0.f), g1 = make_float2(0.f, 0.f);
          if (r < rn) g0 = make_float2(fe0 * m0.x, fe0 * m0.y);
          if (r + 1 < rn) g1 = make_float2(fe1 * m1.x, fe1 * m1.y);
          kt_split_G(Bh, Bl, (uint32_t)boff[i], g0, g1);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(FULL + s));
      }
      cp_async_wait_ahead();  // the next fill's records
      split_dE(t + 1);
      if (named_any(1, KT_PRODN, !ok || *ab)) break;  // one decision for all producers
      rc += KT_RC;
      skip_empty(kc, rc, cc);
    }
    cp_async_wait_all();  // no copy in flight at exit
  } else {
    // ================= epilogue =================
    setmaxnreg_inc<KT_REG_EPI>();
    const int quarter = warp & 3, half = warp >> 2;
    const int nh = N / 2, n8 = nh / 8;  // this warp's columns [half nh, (half + 1) nh), pieces of 8
    const uint32_t D0 = tbase + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(half * nh);
    float* fl = reinterpret_cast<float*>(smk + KT_NST * KT_STAGE + KT_NREC * KT_REC_BYTES + warp * KT_FLUSH_BYTES);
    wbg_u64* bad = out + 4 * (long long)nEF * nOmega * NC;
    constexpr int NP = KT_CT / 8, PB = 3;  // pieces of 8 columns, pieces per batch of loads
    float acc[NP][8];
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[p][i] = 0.f;
    int t = 0;  // fill sequence number
    bool stop = false;
    for (long long k = k0; k < k1 && !stop; ++k) {
      const int nrec = count[k];
      for (int r0 = 0; r0 < nrec; r0 += KT_RC, ++t) {
        const int b = t & 1;
        bool ok = true;
        if (lane == 0) ok = kt_wait(bar(ACCFULL + b), (uint32_t)((t >> 1) & 1), ab, wait_ns);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) {  // a warp-wide decision: the epilogue warps share no barrier after this point
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t D = D0 + (uint32_t)(256 * b);
#pragma unroll
        for (int h = 0; h < NP; h += PB) {
          uint32_t v[PB][8];
#pragma unroll
          for (int p = 0; p < PB; ++p)
            if (h + p < NP && h + p < n8) tmem_ld8(D + 8 * (h + p), v[p]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (h + PB >= NP) {
            tc_fence_before();
            __syncwarp();  // every lane's loads are complete: one arrival per warp frees the accumulator
            if (lane == 0) mbar_arrive(bar(ACCFREE + b));
          }
#pragma unroll
          for (int p = 0; p < PB; ++p)
            if (h + p < NP && h + p < n8) {
              tmem_ld_wait8(v[p]);
#pragma unroll
              for (int i = 0; i < 8; ++i) acc[h + p < NP ? h + p : 0][i] += __uint_as_float(v[p][i]);
            }
        }
      }
      if (!stop && nrec > 0) {  // the k-point's sums into the fixed-point output, two pieces at a time
#pragma unroll
        for (int p = 0; p < NP; p += 2) {
          if (p < n8) {
            float4* f4 = reinterpret_cast<float4*>(fl + lane * KT_FLUSH_LD);
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (p + h < NP) {
                const int ph = p + h < NP ? p + h : 0;
                f4[2 * h] = make_float4(acc[ph][0], acc[ph][1], acc[ph][2], acc[ph][3]);
                f4[2 * h + 1] = make_float4(acc[ph][4], acc[ph][5], acc[ph][6], acc[ph][7]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[ph][i] = 0.f;
              }
            __syncwarp();
            // eight complex columns of four rows per pass
            const int cx = lane & 7, j = (half * nh) / 2 + 4 * p + cx, col = col0 + j;
            const bool act = 4 * p + cx < nh / 2 && j < nct;
            const int e = col / NC, c = col - e * NC;
            for (int i = lane >> 3; i < 32; i += 4) {
              const int w = w0 + 32 * quarter + i;
              if (!act || w >= nOmega) continue;
              const float2 a = *reinterpret_cast<const float2*>(fl + i * KT_FLUSH_LD + 2 * cx);
              wbg_u64* o = out + 4 * (((long long)e * nOmega + w) * NC + c);
              fx_add_double(o, (double)a.x, bad);
              fx_add_double(o + 2, (double)a.y, bad);
            }
            __syncwarp();
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == KT_MMA0 / 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(KT_TMEM_COLS) : "memory");
  }
}
