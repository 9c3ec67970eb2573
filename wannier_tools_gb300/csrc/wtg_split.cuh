// Exactly-split complex products on the 5th-generation tensor cores, shared by
// the mixed form (wtg_mixed.cu) and the FP64 form (wtg_split64.cu).
//
// C = X Y for FP64 complex N x N operands: every operand becomes fixed point
// against a shared exponent per row (left factor) or per column (right factor)
// and is cut into D balanced digits, each an exact 16-bit float; the slice
// products X^p Y^q with p + q <= ORD are MMAs (M = 128 rows, K = 16 a chunk)
// whose FP32 accumulators in tensor memory hold integers of one slice order
// t = p + q, exact while their partial sums stay below 2^24; the accumulators
// are read back, combined as integers and assembled into FP64 with integer
// operations.  Two digit kinds:
//   DigB7  49-bit operands (rounded to nearest) in seven base-128 digits as
//          BF16 (DigB7<4>: the leading four, for corrections); the orders 7
//          and 8 share the last accumulator (they are scaled against each
//          other, which truncates at about 2^-51 of the result)
//   DigF8  55-bit operands (rounded to nearest) in seven base-256 digits as
//          F16; orders 2..9, one exact accumulator each, so a product is as
//          accurate as the rounding of its operands against those exponents
//          (DigF8<4>: the leading four digits and orders 2..5)
//
// Pipeline of one product (split_gemm).  The tiles of the product (row block x
// column pass) are cut into K chunks of 16; the chunks of all tiles form one
// sequence.  Warps 1..15 turn a chunk of both operands into digit planes in
// one of two shared-memory stages and arrive on that stage's `full` barrier;
// one thread of warp 0 issues the chunk's MMAs and commits them to the stage's
// `empty` barrier; no block-wide barrier separates chunks.  The first two
// chunks of the next tile are generated before the accumulators of this one
// are drained, so that the tensor cores restart at once after the drain.  What
// bounds it: the two integer-heavy phases, which take turns at one CTA an SM (the
// pipe is 65-70 % busy in them, 50 % over a launch, and so are the issue slots;
// profiles/k_decimate_split64_arc_n112.md).  At Ndim 112 (F16 digits) a chunk's digit planes
// take 2.8 k cycles against 1.9 k of its MMAs, and 32 columns of accumulators
// 11 k to read back, assemble and store; a product is 142 k cycles (28 chunks,
// 4 tiles; 154 k with the residual's epilogue, 160 k with two FP64 sums).
// Copying the A planes of the first column pass to global memory and loading
// them for the others (bulk copies, 57 KB a chunk) was 5 % slower: they come back
// no faster than they are made.
//
// Digits are made from packed integer extraction and one packed 16-bit
// floating-point FMA per two digits (a digit's bits under a fixed exponent,
// minus the offset: exact).  Generation and drain are mostly integer instructions
// (64 lanes a clock per SM), so both are written for few of them.
//
// Every mbarrier wait is bounded; on a timeout the CTA stops issuing work,
// marks the instance, waits (bounded) for its MMAs and frees tensor memory.
#pragma once

constexpr int SP_T = 512;              // threads per CTA (16 warps)
constexpr int SP_GEN = SP_T - 32;      // digit-generating threads (warps 1..15)
constexpr int KCH = 16;                // K per staged chunk
constexpr int APLANE = 128 * KCH * 2;  // bytes of one A plane (128 rows x 16 digits)
constexpr int MAXD = 7;                // digits per operand
constexpr unsigned SPIN_LIMIT = 1u << 20;
constexpr int PT_TIMEOUT = 8;
constexpr int MX_MAXN = 320;           // largest Ndim
constexpr int MX_SMEM_GJ_N = 112;      // up to here the FP32 Gauss-Jordan runs in shared memory
constexpr int MX_PANEL = 16;           // pivot steps per panel of the global-memory Gauss-Jordan
constexpr int GJS_PANEL = 8;           // and of the shared-memory one
constexpr int MX_ROWS = MX_MAXN / 32;  // rows per lane of a register-resident column
constexpr int EXP_MIN = 80;            // shared exponents are at least this (biased): rows and
                                       // columns below 2^-940 count as zero

constexpr int OZ_STORE = 0, OZ_ADD2 = 1, OZ_STORE_NORM = 2, OZ_IMINUS = 3, OZ_ADDTO = 4;

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: K-major, no swizzle, LBO 128 B (K), SBO 256 B (rows)
__device__ __forceinline__ uint64_t sdesc(uint32_t a) {
  return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) |
         ((uint64_t)(256 >> 4) << 32) | (1ull << 46);
}

// kind::f16 (BF16 or F16 operands by the instruction descriptor), FP32 accumulators
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t id,
                                        uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(id), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint64_t* mb) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   saddr(mb))
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mb) {
  asm volatile("{\n .reg .b64 t;\n mbarrier.arrive.shared::cta.b64 t, [%0];\n}\n" ::"r"(saddr(mb))
               : "memory");
}

// Bounded wait for an mbarrier phase.  limit 0: up to SPIN_LIMIT blocking
// try_wait polls (the normal bound); limit > 0 (a test's bound): that many
// non-blocking test_wait polls, so that a short limit reliably runs out while
// the tensor cores are still busy.
__device__ __forceinline__ bool mbar_wait(uint64_t* mb, uint32_t parity, unsigned limit = 0) {
  const uint32_t a = saddr(mb);
  if (limit == 0) {
    for (unsigned spin = 0; spin < SPIN_LIMIT; ++spin) {
      uint32_t ok;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(ok)
          : "r"(a), "r"(parity)
          : "memory");
      if (ok) return true;
    }
    return false;
  }
  for (unsigned spin = 0; spin < limit; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- integer-only conversions ---------------------------------------------

__device__ __forceinline__ int bexp(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF);
}

// logical right shift by any amount (64 and above give 0)
__device__ __forceinline__ unsigned long long shr64(unsigned long long v, unsigned n) {
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
  return r;
}

// 53-bit significand of a normal x with its hidden bit (the shift that follows
// drops a denormal's whole, as its shared exponent is at least EXP_MIN)
__device__ __forceinline__ unsigned long long signif(unsigned long long u) {
  return (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
}

// double with value S * 2^(be0 - 1023) assembled from bits, without branches;
// ROUND: to nearest (ties away), otherwise truncating.  Results below the normal
// range are 0.
template <bool ROUND>
__device__ __forceinline__ double assemble(long long S, int be0) {
  const long long sg = S >> 63;
  const unsigned long long a = (unsigned long long)((S ^ sg) - sg);
  const int lz = __clzll((long long)a);
  const unsigned long long n = a << (lz & 63);        // leading bit at 63
  const int be = 63 - lz + be0;
  unsigned long long m = n >> 11;                     // the hidden bit adds 1 to the exponent
  if (ROUND) m += (n >> 10) & 1ull;
  unsigned long long r = ((unsigned long long)(unsigned)(be - 1) << 52) + m;
  r = be >= 2047 ? 0x7FF0000000000000ull : r;
  r = (be <= 0 || a == 0) ? 0ull : r;
  return __longlong_as_double((long long)(r | ((unsigned long long)sg << 63)));
}

// a b + c, one instruction of the multiply pipe
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  return (long long)a * b + c;
}

// assemble for |S| < 2^63, with the common case (zero, or |S| >= 2^32 and a normal
// result) in about half the instructions: the drain of the accumulators is
// bound by the integer pipe
template <bool ROUND>
__device__ __forceinline__ double assemble_fast(long long S, int be0) {
  const long long sg = S >> 63;
  const unsigned long long a = (unsigned long long)((S ^ sg) - sg);
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
  const int lz = __clz((int)ah);                      // 1..31, or 32 (zero, or below 2^32)
  const unsigned be1 = (unsigned)(62 - lz + be0);
  if (ah == 0 ? al != 0 : be1 >= 2045u) return assemble<ROUND>(S, be0);
  // leading bit at 62: two 32-bit shifts
  unsigned long long n =
      ((unsigned long long)__funnelshift_l(al, ah, (unsigned)lz - 1) << 32) | (al << ((lz - 1) & 31));
  if (ROUND) n += 0x200;
  const unsigned long long m = n >> 10;               // the hidden bit adds 1 to the exponent
  const unsigned hi = ((unsigned)(m >> 32) + (be1 << 20)) | ((unsigned)(S >> 32) & 0x80000000u);
  return __hiloint2double((int)(ah ? hi : 0u), (int)(unsigned)m);
}

__device__ __forceinline__ double f2d_bits(float f) {     // exact FP32 -> FP64
  const uint32_t w = __float_as_uint(f);
  const unsigned long long sign = (unsigned long long)(w >> 31) << 63;
  const int e = (int)((w >> 23) & 0xFF);
  if (e == 0) return __longlong_as_double((long long)sign);
  if (e == 255) return __longlong_as_double((long long)(sign | (0x7FFull << 52)));
  return __longlong_as_double(
      (long long)(sign | ((unsigned long long)(e - 127 + 1023) << 52) |
                  ((unsigned long long)(w & 0x7FFFFFu) << 29)));
}

// ---- digit kinds -------------------------------------------------------------

// packed 16-bit floating point on raw words
__device__ __forceinline__ uint32_t hfma2_f16(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t hfma2_bf16(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// Base-128 digits as BF16.  |x| = f 2^(E - 1022 - 49), f < 2^49 rounded to
// nearest (ties up); f + 64 (1 + 128 + .. + 128^5) has digits g_p in [0, 127]
// below the leading one (in [0, 128]), and f = sum of (g_p - 64) 128^(7-p) with
// the leading digit as it stands.  A BF16 word 0x4300 | g is 128 + g, so that
// (128 + g) 2^s - (128 + 64) 2^s is the digit times its power of two, exactly,
// by one packed FMA; the element's sign is XORed in.
template <int D_>
struct DigB7 {
  static constexpr int D = D_;
  static constexpr int ORD = D == 7 ? 8 : 5;          // slice pairs p + q <= ORD
  static constexpr int NACC = D == 7 ? 6 : 4;         // orders 2..; the last one lumped at D = 7
  static constexpr bool LUMPED = D == 7;
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
  static constexpr int KSPLIT = 1 << 20;              // K of one exact accumulation
  static constexpr bool POISON = false;
  static constexpr bool FRO = false;
  static constexpr int SLOT = D == 7 ? 0 : 2;         // its issue tables (full and last width)

  static constexpr unsigned long long BIAS =
      64ull * (1ull + (1ull << 7) + (1ull << 14) + (1ull << 21) + (1ull << 28) + (1ull << 35));
  struct Fix {
    uint32_t lo, hi;                                  // 2 (f + BIAS) + rounding bit
  };
  static __device__ __forceinline__ Fix fix(double x, int E) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(u >> 52) & 0x7FF;
    const unsigned long long t = shr64(signif(u), (unsigned)(E - ex + 3)) + (1 + 2 * BIAS);
    return Fix{(uint32_t)t, (uint32_t)(t >> 32)};
  }
  static __host__ __device__ constexpr uint32_t two(uint32_t h) { return h | (h << 16); }
  // 2^s, and -(128 + bias) 2^s, as BF16 pairs
  static __host__ __device__ constexpr uint32_t scale(int s) { return two((uint32_t)(127 + s) << 7); }
  static __host__ __device__ constexpr uint32_t offset(int s, bool lead) {
    return two(0x8000u | ((uint32_t)(134 + s) << 7) | (lead ? 0u : 0x40u));
  }
  template <int P, int E0>
  static __device__ __forceinline__ uint32_t digit(const Fix& a, const Fix& b, uint32_t sgn) {
    constexpr int SH = P == 1 ? 43 : P <= 3 ? 29 : P <= 5 ? 15 : 1;   // 14-bit groups of 2 f
    uint32_t g;
    if constexpr (SH == 43) {
      g = __byte_perm(a.hi >> 11, b.hi >> 11, 0x5410);
    } else {
      g = __byte_perm(__funnelshift_r(a.lo, a.hi, SH), __funnelshift_r(b.lo, b.hi, SH), 0x5410);
      if constexpr ((P & 1) == 0) g >>= 7;
    }
    g = (g & (P == 1 ? 0x00FF00FFu : 0x007F007Fu)) | 0x43004300u;
    constexpr int s = 7 * (E0 - P);
    return hfma2_bf16(g, scale(s), offset(s, P == 1)) ^ sgn;
  }
  // the D digit words of a pair of reals (elements k and k + 1)
  template <int E0>
  static __device__ __forceinline__ void digits(double x0, double x1, int E, uint32_t (&w)[D]) {
    const Fix a = fix(x0, E), b = fix(x1, E);
    const uint32_t sgn = ((uint32_t)__double2hiint(x0) >> 31 << 15) |
                         ((uint32_t)__double2hiint(x1) & 0x80000000u);
    w[0] = digit<1, E0>(a, b, sgn);
    w[1] = digit<2, E0>(a, b, sgn);
    w[2] = digit<3, E0>(a, b, sgn);
    w[3] = digit<4, E0>(a, b, sgn);
    if constexpr (D > 4) {
      w[4] = digit<5, E0>(a, b, sgn);
      w[5] = digit<6, E0>(a, b, sgn);
      w[6] = digit<7, E0>(a, b, sgn);
    }
  }
  static __device__ __forceinline__ void digits_a(double x0, double x1, int E, uint32_t (&w)[D]) {
    digits<3>(x0, x1, E, w);
  }
  static __device__ __forceinline__ void digits_b(double x0, double x1, int E, uint32_t (&w)[D]) {
    digits<5>(x0, x1, E, w);
  }
  static __device__ __forceinline__ void digits_pm(double x0, double x1, int E, uint32_t (&w)[D],
                                                   uint32_t (&wn)[D]) {
    digits<5>(x0, x1, E, w);
#pragma unroll
    for (int p = 0; p < D; ++p) wn[p] = w[p] ^ 0x80008000u;
  }
  template <int T>
  static __device__ __forceinline__ int m_of(uint32_t v) {
    return __float2int_rz(__uint_as_float(v) * __int_as_float((127 + 7 * T - 56) << 23));
  }
  // value of the accumulators of one output component
  static __device__ __forceinline__ double value(const uint32_t (&v)[NACC], int ee) {
    // exact order t: the accumulator is m 2^(56-7t), |m| < 2^24; the orders >= 7
    // are taken in units of 2^7, truncated
    long long S = LUMPED ? (long long)m_of<7>(v[NACC - 1]) : 0;
#pragma unroll
    for (int a = 0; a < NACC - (LUMPED ? 1 : 0); ++a) {
      const int m = a == 0 ? m_of<2>(v[0]) : a == 1 ? m_of<3>(v[1]) : a == 2 ? m_of<4>(v[2])
                    : a == 3 ? m_of<5>(v[3]) : m_of<6>(v[a]);
      S += a == 0 ? (long long)((unsigned long long)(long long)m << 35)
                  : (long long)m * (1ll << (49 - 7 * (a + 2)));
    }
    return assemble_fast<false>(S, ee - 1070);
  }
};

// Base-256 digits as F16.  |x| = F 2^(E - 1022 - 54), F <= 2^54 rounded to
// nearest; F + 128 (1 + 256 + .. + 256^6) has byte digits g_p, and F = sum of
// (g_p - 128) 256^(7-p): the leading digit is in [0, 64], the others in
// [-128, 127].  An F16 word 0x6400 | g is 1024 + g, so (1024 + g) s - 1152 s is
// the digit times the element's sign s, exactly, by one packed FMA.  Order t gathers 2 (t - 1) K
// digit products of at most 2^12 (1, 1), 2^13 (1, q) or 2^14: below 2^24 for
// the orders 2..5 at K <= 170 and order 6 at K <= 128 even with every product
// at its bound and of one sign; above that, K is accumulated in parts of at
// most 160 (KSPLIT), and an order >= 6 that passed 2^24 in such a case would
// lose a unit of 2^-44 or less, where an FP64 product's own bound is 2K 2^-53.
// The orders above 9 (at most 2^-58 of the row and column scales a term) are
// dropped.
template <int D_>
struct DigF8 {
  static constexpr int D = D_;
  static constexpr int ORD = D == 7 ? 9 : 5;
  static constexpr int NACC = ORD - 1;
  static constexpr bool LUMPED = false;
  static constexpr uint32_t IDESC = (1u << 4) | ((128u >> 4) << 24);
  static constexpr int KSPLIT = 160;
  static constexpr int SLOT = D == 7 ? 0 : 2;
  static constexpr bool FRO = true;
  static constexpr bool POISON = true;                // Inf / NaN in a row or column give NaN

  static constexpr unsigned long long BIAS = 0x80808080808080ull;
  struct Fix {
    uint32_t lo, hi;                                  // bytes g_7 .. g_4 | g_3 g_2 g_1 0x64
  };
  // |x|: (((|x| 2^(55 - E + 1022)) truncated) + 1) / 2 = |F|
  static __device__ __forceinline__ Fix fix(double x, int E) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(u >> 52) & 0x7FF;
    const unsigned long long v =
        (shr64(signif(u) << 2, (unsigned)(E - ex)) + (1 + 2 * BIAS + (0x64ull << 57))) >> 1;
    return Fix{(uint32_t)v, (uint32_t)(v >> 32)};
  }
  template <int P>
  static __device__ __forceinline__ uint32_t biased(const Fix& a, const Fix& b) {
    if constexpr (P <= 3) {
      constexpr uint32_t j = 3 - P;
      return __byte_perm(a.hi, b.hi, j | 0x30u | ((4 + j) << 8) | 0x7000u);
    } else {
      constexpr uint32_t j = 7 - P;
      return (__byte_perm(a.lo, b.lo, j | (j << 4) | ((4 + j) << 8) | ((4 + j) << 12)) &
              0x00FF00FFu) | 0x64006400u;
    }
  }
  // the D digit words of a pair of reals and, with NEG, their negatives
  template <bool NEG>
  static __device__ __forceinline__ void digits(double x0, double x1, int E, uint32_t (&w)[D],
                                                uint32_t (&wn)[D]) {
    const Fix a = fix(x0, E), b = fix(x1, E);
    uint32_t g[D];
    g[0] = biased<1>(a, b);
    g[1] = biased<2>(a, b);
    g[2] = biased<3>(a, b);
    g[3] = biased<4>(a, b);
    if constexpr (D > 4) {
      g[4] = biased<5>(a, b);
      g[5] = biased<6>(a, b);
      g[6] = biased<7>(a, b);
    }
    // +-1 and -+1152 by the elements' signs, as F16 pairs
    const uint32_t sg = __byte_perm((uint32_t)__double2hiint(x0), (uint32_t)__double2hiint(x1), 0x7632) &
                        0x80008000u;
    const uint32_t one = sg | 0x3C003C00u, off = sg ^ 0xE480E480u;
#pragma unroll
    for (int p = 0; p < D; ++p) {
      w[p] = hfma2_f16(g[p], one, off);
      if (NEG) wn[p] = hfma2_f16(g[p], one ^ 0x80008000u, off ^ 0x80008000u);
    }
  }
  static __device__ __forceinline__ void digits_a(double x0, double x1, int E, uint32_t (&w)[D]) {
    digits<false>(x0, x1, E, w, w);
  }
  static __device__ __forceinline__ void digits_b(double x0, double x1, int E, uint32_t (&w)[D]) {
    digits<false>(x0, x1, E, w, w);
  }
  static __device__ __forceinline__ void digits_pm(double x0, double x1, int E, uint32_t (&w)[D],
                                                   uint32_t (&wn)[D]) {
    digits<true>(x0, x1, E, w, wn);
  }
  static __device__ __forceinline__ int f2i(uint32_t v) {
    return __float2int_rz(__uint_as_float(v));
  }
  // value of the accumulators of one output component
  static __device__ __forceinline__ double value(const uint32_t (&v)[NACC], int ee) {
    // order t in units of 256^(14-t) 2^(ee - 2152)
    if constexpr (D > 4) {
      // the sum in units of 256^5 2^14, a quarter of order 7's: |sum| < 2^63.  The orders
      // 7..9 are added in FP32 (2^-24 of order 7, at most 2^-58 of the scales for
      // partial sums of random digits) and converted together; order 2, below
      // 2^22, is converted by an add (conversions run at 16 a clock per SM)
      const float f789 = fmaf(__uint_as_float(v[7]), 0x1p-14f,
                              fmaf(__uint_as_float(v[6]), 0x1p-6f, 4.0f * __uint_as_float(v[5])));
      const int low = __float2int_rn(f789);
      const int m2 = __float_as_int(__uint_as_float(v[0]) + 12582912.0f);      // + 0x4B400000
      const long long S = mad_wide(f2i(v[2]), 1 << 26,
                                   mad_wide(f2i(v[3]), 1 << 18, mad_wide(f2i(v[4]), 1 << 10, low)));
      const unsigned top = (unsigned)m2 * 1024u + ((unsigned)f2i(v[1]) * 4u);  // in units of 2^32
      return assemble_fast<true>(S + (long long)((unsigned long long)top << 32),
                                 ee - 2152 + 54 + 1023);
    } else {
      const long long S = mad_wide(f2i(v[0]), 1 << 24,
                                   mad_wide(f2i(v[1]), 1 << 16, mad_wide(f2i(v[2]), 1 << 8, f2i(v[3]))));
      return assemble_fast<true>(S, ee - 2152 + 72 + 1023);
    }
  }
};

// ---- passes and shared memory ------------------------------------------------

// How the output columns of a product are cut into tensor-memory passes:
// columns [0, NP) in blocks of w0 (a multiple of 8; the last one narrower).  A
// pass holds NACC accumulators of 2 w0 columns (both components side by side)
// in the 512 tensor-memory columns.
struct MxPlan {
  int N, NP, nrb, ncb, w0;
  int wb;                    // B-plane width of the shared-memory layout (7-digit stages)
};

template <class K>
__host__ __device__ constexpr int split_wmax() {
  return (512 / (2 * K::NACC)) & ~7;
}

// w0_req: a pass width from the tile table (a multiple of 8 in [8, wmax]); any
// other value takes the built-in choice (the fewest passes, evenly split)
__host__ __device__ inline MxPlan split_plan(int N, int wmax, int w0_req = 0) {
  MxPlan p;
  p.N = N;
  p.NP = (N + 7) & ~7;          // an MMA's N (2w, both components) needs w a multiple of 8 only
  p.nrb = (N + 127) / 128;
  if (w0_req >= 8 && w0_req <= wmax && (w0_req & 7) == 0) {
    p.w0 = w0_req;
    p.ncb = (p.NP + w0_req - 1) / w0_req;
  } else {
    p.ncb = (p.NP + wmax - 1) / wmax;
    p.w0 = ((p.NP + p.ncb - 1) / p.ncb + 7) & ~7;
    while (p.ncb > 1 && (p.ncb - 1) * p.w0 >= p.NP) --p.ncb;
  }
  p.wb = p.w0;
  return p;
}

// the plan of a 4-digit product in the stages of a 7-digit one: as wide as the
// tensor memory (four accumulators) and the stage's B area allow
__host__ __device__ inline MxPlan split_plan4(const MxPlan& p7) {
  int wmax = (512 / (2 * 4)) & ~7;
  const int bcap = ((4 * MAXD * p7.wb) / (4 * 4)) & ~7;
  if (bcap < wmax) wmax = bcap;
  MxPlan p = split_plan(p7.N, wmax);
  p.wb = p7.wb;
  return p;
}

// issue tables of a chunk's MMAs (issue_table)
constexpr int TAB_MAX = 40;
struct IssueTab {
  uint4 e[TAB_MAX];
};

__host__ __device__ __forceinline__ int stage_bytes_of(int WB) {
  return 2 * MAXD * APLANE + 4 * MAXD * WB * KCH * 2;
}

// Bytes of the FP64 Gauss-Jordan working area (fp64_layout with KC = GJ_PANEL):
// the N x N matrix and its small arrays when the inverse runs in shared memory,
// the panel arrays when it runs in global memory.
__host__ __device__ constexpr int fp64_area_bytes(int N, bool in_smem) {
  return (in_smem ? (N * N > 2 * N * GJ_PANEL ? N * N : 2 * N * GJ_PANEL) : 2 * N * GJ_PANEL) * 16 +
         N * 32 + 16 * GJ_PANEL + 32 * 8 + N * 8 + 16;
}
// the largest over Ndim 1..MX_MAXN (shared-memory inverse up to MX_SMEM_GJ_N)
constexpr int MX_FP64_AREA =
    fp64_area_bytes(MX_SMEM_GJ_N, true) > fp64_area_bytes(MX_MAXN, false)
        ? fp64_area_bytes(MX_SMEM_GJ_N, true) : fp64_area_bytes(MX_MAXN, false);

// bytes before the small arrays: the two operand stages and the exponents of
// the workspace matrices, which the FP64 inverse area aliases (the FP32
// Gauss-Jordan matrix or its panel multipliers alias the stages only)
constexpr int EXPS_BYTES = 8 * 2 * MX_MAXN * 4;
__host__ __device__ __forceinline__ int planes_bytes_of(int WB) {
  const int two = 2 * stage_bytes_of(WB) + EXPS_BYTES;
  return ((two > MX_FP64_AREA ? two : MX_FP64_AREA) + 1023) & ~1023;
}
// small arrays, at their byte offsets behind that region
struct SplitTail {
  float2 recip[MX_PANEL];
  int prow[MX_MAXN];             // Gauss-Jordan: pivot rows
  int pos_of[MX_MAXN];           // Gauss-Jordan: position of a row, row at a position
  int row_at[MX_MAXN];
  IssueTab tabs[4];              // a 7-digit product's full and last pass width, then a 4-digit one's
  int ntab[4];
  float red[32];
  uint64_t full[2];              // a stage's digits are complete (one arrival per generating warp)
  uint64_t empty[2];             // a stage's MMAs are complete
  uint32_t tslot;                // tensor-memory address
  uint32_t chunk;                // chunks generated so far (a chunk's stage is its low bit)
  uint32_t issued;               // chunks committed
  int abort;                     // a wait gave up
  unsigned spin;                 // pipeline waits' bound (0 = built-in; see mbar_wait)
  int misc[5];                   // 0 instance, 1 singular, 2-3 pivot rows (shared-memory Gauss-Jordan)
};
constexpr int SPLIT_TAIL = (int)sizeof(SplitTail);
static_assert(2 * GJS_PANEL <= MX_PANEL, "two panels' multipliers and reciprocals");
// the FP32 Gauss-Jordan areas (matrix and multipliers) fit below the exponents for
// every stage width
static_assert((MX_SMEM_GJ_N + MX_PANEL) * MX_SMEM_GJ_N * 8 <= 2 * 2 * MAXD * APLANE, "FP32 GJ area");
static_assert(MX_MAXN * MX_PANEL * 8 <= 2 * 2 * MAXD * APLANE, "FP32 GJ panel area");

__host__ __device__ __forceinline__ size_t split_smem(int WB) {
  return (size_t)planes_bytes_of(WB) + SPLIT_TAIL;
}

// Shared-memory layout: two operand stages (2 MAXD A planes, then 4 MAXD B
// planes of wb rows each), the exponents, then the small arrays.  Two integers
// and the shared array itself, so that it lives in registers and every access
// compiles to a shared-memory instruction: beside 217 KB of shared memory the
// L1 holds a few tens of KB, so a stack frame or a spill of 512 threads is
// served by the L2 (pointers kept in a structure on the stack made every step
// of the accumulator drain several times slower).
struct MxShared {
  int stage, tail;
  static __device__ __forceinline__ unsigned char* base() {
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    return smem_dyn;
  }
  __device__ __forceinline__ SplitTail& t() const {
    return *reinterpret_cast<SplitTail*>(base() + tail);
  }
  // row exponents of workspace matrix i (0..10; matrices 3..10 have them), then
  // its column exponents
  __device__ __forceinline__ int* rows(int i, int N) const {
    return reinterpret_cast<int*>(base() + 2 * stage) + 2 * N * (i & 7);
  }
  __device__ __forceinline__ int* cols(int i, int N) const { return rows(i, N) + N; }
};
__device__ __forceinline__ MxShared mx_layout(int WB) {
  return MxShared{stage_bytes_of(WB), planes_bytes_of(WB)};
}

// row and column exponents of workspace matrix i by a pass over it (all threads;
// ends with a barrier)
__device__ __noinline__ void exps_of(const double2* __restrict__ p, int i, int N, MxShared s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  int* const er = s.rows(i, N);
  int* const ec = s.cols(i, N);
  for (int r = threadIdx.x; r < N; r += blockDim.x) er[r] = EXP_MIN;
  __syncthreads();
  int rmax[MX_ROWS];
#pragma unroll
  for (int q = 0; q < MX_ROWS; ++q) rmax[q] = 0;
  for (int j = warp; j < N; j += nwarp) {
    const double2* col = p + (size_t)j * N;
    int c = EXP_MIN;
#pragma unroll
    for (int q = 0; q < MX_ROWS; ++q) {
      const int r = lane + 32 * q;
      if (r < N) {
        const double2 v = col[r];
        const int e = max(bexp(v.x), bexp(v.y));
        rmax[q] = max(rmax[q], e);
        c = max(c, e);
      }
    }
    c = __reduce_max_sync(0xffffffffu, c);
    if (lane == 0) ec[j] = c;
  }
#pragma unroll
  for (int q = 0; q < MX_ROWS; ++q)
    if (lane + 32 * q < N) atomicMax(&er[lane + 32 * q], rmax[q]);
  __syncthreads();
}

// ---- the product -------------------------------------------------------------

// The MMAs of one chunk as a table: one entry per group of slice pairs (two
// MMAs).  The B digit planes are stored in two runs, Yr, Yi of digit q at planes
// 2(q-1), +1 and -Yi, Yr at 2D + 2(q-1), +1, so that [Yr; Yi] and [-Yi; Yr] of g
// consecutive digits are each one operand of 2wg rows: Xr [Yr; Yi] and
// Xi [-Yi; Yr] accumulate [Cr | Ci].  Slice order t goes to accumulator
// min(t - 2, NACC - 1); accumulator a sits at tensor-memory column 2 w a.  For
// one digit p of X, the pairs of g consecutive digits q whose orders have
// consecutive accumulators are one MMA of N = 2 w g <= 256; the first MMA into
// an accumulator overwrites, so a group's accumulators are all new or all
// written.  An entry: offsets of the A and B planes in descriptor units (16 B),
// tensor-memory column (bit 31: new accumulators), instruction descriptor.
// Why a table: tcgen05.mma runs N / 2 cycles (M = 128, K = 16; N >= 96) when the
// issuing thread keeps up, but a thread that works out each MMA's operands
// first issues one per 250 cycles.
template <class K>
__device__ void issue_table(IssueTab* tab, int* count, int width) {
  constexpr int D = K::D, NEX = K::NACC - (K::LUMPED ? 1 : 0);
  const uint32_t bplane16 = (uint32_t)width * KCH * 2 >> 4;
  const int gmax = 128 / width;                  // 2 w g <= 256 columns
  uint32_t amask = 0u;
  int n = 0;
  for (int p = 1; p <= D; ++p) {
    const int qn = min(D, K::ORD - p);
    int q = 1;
    while (q <= qn) {
      const int t0 = p + q;
      const int a0 = t0 - 2 < NEX ? t0 - 2 : K::NACC - 1;
      const uint32_t touched = (amask >> a0) & 1u;
      int g = 1;
      while (g < gmax && q + g <= qn) {
        const int t = t0 + g;
        const int a = t - 2 < NEX ? t - 2 : K::NACC - 1;
        if (a != a0 + g || ((amask >> a) & 1u) != touched) break;
        ++g;
      }
      amask |= ((1u << g) - 1u) << a0;
      if (n < TAB_MAX)
        tab->e[n] = make_uint4((uint32_t)(2 * (p - 1)) * (APLANE >> 4),
                               (uint32_t)(2 * (q - 1)) * bplane16,
                               (uint32_t)(a0 * 2 * width) | (touched ? 0u : 0x80000000u),
                               K::IDESC | ((uint32_t)(2 * width * g >> 3) << 17));
      ++n;
      q += g;
    }
  }
  *count = n;
}

// one chunk's MMAs from stage A (one elected thread; later: not the tile's first chunk)
template <class K>
__device__ __forceinline__ void split_issue(const IssueTab* tab, int n, uint32_t A, uint32_t tmem,
                                            int width, bool later) {
  const uint64_t a0 = sdesc(A), b0 = sdesc(A + 2 * MAXD * APLANE);
  const uint64_t neg = (uint64_t)(2 * K::D) * ((uint32_t)width * KCH * 2 >> 4);
#pragma unroll 4
  for (int i = 0; i < n; ++i) {
    const uint4 e = tab->e[i];
    const uint32_t d = tmem + (e.z & 0xFFFFu);
    mma_f16(d, a0 + e.x, b0 + e.y, e.w, (later || !(e.z >> 31)) ? 1u : 0u);
    mma_f16(d, a0 + e.x + (APLANE >> 4), b0 + e.y + neg, e.w, 1u);
  }
}

// one thread of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}

// |re + i im| in FP64 (Fortran's abs of a complex(dp)); hypot's scaling only
// outside the range where the squares neither overflow nor underflow
__device__ __forceinline__ double cabs64(double re, double im) {
  const double a = fabs(re), b = fabs(im), h = fmax(a, b);
  if (h < 0x1p500 && h > 0x1p-500) return sqrt(fma(a, a, b * b));
  return h == 0.0 ? 0.0 : hypot(a, b);
}

// One product's operands and outputs as workspace matrix indices: X, Y, out0
// and aux (OZ_ADD2: the second sum; OZ_ADDTO: the addend), and the lower rows'
// X, out0 and aux of a stacked product.  Outputs at index 3 and above get their
// exponents.
__host__ __device__ constexpr uint32_t ops(int X, int Y, int out, int aux = 0, int Xl = 0,
                                           int outl = 0, int auxl = 0) {
  return (uint32_t)(X | (Y << 4) | (out << 8) | (aux << 12) | (Xl << 16) | (outl << 20) |
                    (auxl << 24));
}

// One work item of a chunk: a pair of K-adjacent elements of one row of X (A
// planes) or of one column of Y (B planes).  In the canonical layout item `it`
// covers row 8 (it >> 6) + ((it & 31) >> 2) and K pair 8 ((it >> 5) & 1) +
// 2 (it & 3), and its word sits at byte 4 it of a plane: each warp store fills
// one 128-byte core matrix (no bank conflicts), each warp load 8 rows x 8 k.
__device__ __forceinline__ int item_row(int it) { return (it >> 6) * 8 + ((it & 31) >> 2); }
__device__ __forceinline__ int item_k(int it) { return ((it >> 5) & 1) * 8 + (it & 3) * 2; }

// A tile of a product: a row block of 128, a column pass and a part of K; its
// chunks are 16 of K.  next() steps through a product's tiles (K part fastest,
// then the pass, then the row block) without divisions: a product at Ndim 40 has
// two tiles of three chunks, and the position arithmetic was a tenth of it.
struct Tile {
  int rb0, jb, width, ka, kb;
  __device__ __forceinline__ int chunks() const { return (kb - ka + KCH - 1) / KCH; }
};
template <class K>
__device__ __forceinline__ int k_part(int N) {       // K of one part
  const int nks = (N + K::KSPLIT - 1) / K::KSPLIT;
  return nks <= 1 ? N : (((N + nks - 1) / nks + KCH - 1) & ~(KCH - 1));
}
__device__ __forceinline__ Tile first_tile(int N, int NP, int w0, int kper) {
  return Tile{0, 0, min(w0, NP), 0, min(N, kper)};
}
// false: t was the last tile (it is left as it is)
__device__ __forceinline__ bool next_tile(Tile& t, int M, int N, int NP, int w0, int kper) {
  if (t.kb < N) {
    t.ka = t.kb;
    t.kb = min(N, t.kb + kper);
    return true;
  }
  if (t.jb + w0 < NP) {
    t.jb += w0;
  } else {
    if (t.rb0 + 128 >= M) return false;
    t.rb0 += 128;
    t.jb = 0;
  }
  t.width = min(w0, NP - t.jb);
  t.ka = 0;
  t.kb = min(N, kper);
  return true;
}

// Digit planes of a tile's chunks gc .. ge-1 (warps 1..15), chunk gc being
// number `chunk` of the kernel's chunk sequence.  Returns 1 when a wait gave up.
// A function of its own (as split_drain), so that neither phase's registers are
// live in the other: one function for both spilled.
template <class K>
__device__ __noinline__ int split_generate(const double2* __restrict__ W, uint32_t op, int N,
                                           int M, Tile T, int gc, int ge, uint32_t chunk,
                                           MxShared s) {
  constexpr int D = K::D;
  constexpr int NR = D == 7 ? 3 : 4;             // rounds of items per generating thread
  SplitTail& sh = s.t();
  const int NN = N * N;
  const int gtid = threadIdx.x - 32, lane = threadIdx.x & 31;
  const int width = T.width, ka = T.ka, kb = T.kb;
  // this thread's items: element address at chunk gc, distance of the pair's
  // second element, shared exponent (address null: zeros)
  const double2* px[NR];
  int ex[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int it = gtid + r * SP_GEN;
    px[r] = nullptr;
    ex[r] = EXP_MIN;
    const int k = ka + gc * KCH + item_k(it);    // 1024 is a multiple of 64: the same for B items
    if (it < 1024) {
      const int i = T.rb0 + item_row(it);
      if (i < M) {
        const bool low = i >= N;                 // the second product's rows of a stacked pair
        const int m = low ? (op >> 16) & 15 : op & 15, il = low ? i - N : i;
        px[r] = W + (size_t)(m * NN) + il + k * N;
        ex[r] = s.rows(m, N)[il];
      }
    } else if (it - 1024 < width * 8) {
      const int j = T.jb + item_row(it - 1024), m = (op >> 4) & 15;
      if (j < N) {
        px[r] = W + (size_t)(m * NN) + j * N + k;
        ex[r] = s.cols(m, N)[j];
      }
    }
  }
  double2 raw[NR][2];
  auto load = [&](int c) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int it = gtid + r * SP_GEN;
      const int k = ka + c * KCH + item_k(it);
      raw[r][0] = make_double2(0.0, 0.0);
      raw[r][1] = raw[r][0];
      if (px[r]) {
        if (k < kb) raw[r][0] = *px[r];
        if (k + 1 < kb) raw[r][1] = px[r][it < 1024 ? N : 1];
        px[r] += it < 1024 ? KCH * N : KCH;
      }
    }
  };
  load(gc);
  for (int c = gc; c < ge; ++c, ++chunk) {
    const int b = chunk & 1;
    const bool ok = chunk < 2 || mbar_wait(&sh.empty[b], ((chunk >> 1) - 1) & 1, sh.spin);
    if (!__all_sync(0xffffffffu, ok)) return 1;
    unsigned char* const A = s.base() + b * s.stage;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int it = gtid + r * SP_GEN;
      uint32_t w[D];
      if (it < 1024) {
        uint32_t* const dst = reinterpret_cast<uint32_t*>(A) + it;
        if (__all_sync(0xffffffffu, px[r] == nullptr)) {     // 8 padding rows of the tile
#pragma unroll
          for (int p = 0; p < 2 * D; ++p) dst[p * (APLANE / 4)] = 0u;
          continue;
        }
        K::digits_a(raw[r][0].x, raw[r][1].x, ex[r], w);
#pragma unroll
        for (int p = 0; p < D; ++p) dst[2 * p * (APLANE / 4)] = w[p];
        K::digits_a(raw[r][0].y, raw[r][1].y, ex[r], w);
#pragma unroll
        for (int p = 0; p < D; ++p) dst[(2 * p + 1) * (APLANE / 4)] = w[p];
      } else if (it - 1024 < width * 8) {
        uint32_t* const dst = reinterpret_cast<uint32_t*>(A + 2 * MAXD * APLANE) + (it - 1024);
        // running addresses: Yr planes and, 2D planes further, -Yi, Yr
        const int bs = width * KCH * 2 / 4;      // B plane stride in words
        K::digits_b(raw[r][0].x, raw[r][1].x, ex[r], w);
        uint32_t* d0 = dst;
        uint32_t* d1 = dst + (2 * D + 1) * bs;
#pragma unroll
        for (int p = 0; p < D; ++p, d0 += 2 * bs, d1 += 2 * bs) {
          *d0 = w[p];
          *d1 = w[p];
        }
        uint32_t wn[D];
        K::digits_pm(raw[r][0].y, raw[r][1].y, ex[r], w, wn);
        d0 = dst + bs;
        d1 = dst + 2 * D * bs;
#pragma unroll
        for (int p = 0; p < D; ++p, d0 += 2 * bs, d1 += 2 * bs) {
          *d0 = w[p];
          *d1 = wn[p];
        }
      }
    }
    if (c + 1 < ge) load(c + 1);                 // before the wait for its stage
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.full[b]);
  }
  return 0;
}

// a - b where it stands: not computed ahead of the branch around it (two FP64
// operations a clock: speculated subtractions cost a tenth of a product)
__device__ __forceinline__ double dsub_here(double a, double b) {
  double r;
  asm volatile("sub.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}

// |x| from its upper word: the magnitude truncated to 21 bits, 0 or Inf outside
// FP32's range (the sums it goes into are compared with margins far above 2^-20)
__device__ __forceinline__ float upper_f32(double x) {
  const int h = (__double2hiint(x) & 0x7FFFFFFF) - (896 << 20);
  return __int_as_float(min(max(h, 0), 0x0FF00000) << 3);
}

// Accumulators of a tile through the epilogue (all warps: four per quadrant of
// 32 tensor-memory lanes, each taking 2 of every 8 columns).  Returns this
// thread's part of the product's FP32 sum.
template <class K>
__device__ __noinline__ float split_drain(double2* __restrict__ W, uint32_t op, int EPI, int EPI2,
                                          int N, int M, Tile T, float nrm, MxShared s) {
  constexpr int NACC = K::NACC;
  const bool STACK = EPI2 >= 0;
  const size_t NN = (size_t)N * N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rb0 = T.rb0, jb = T.jb, width = T.width;
  const bool first = T.ka == 0, last = T.kb == N;
  const int quad = warp & 3, hw = warp >> 2;
  // a warp whose 32 tensor-memory lanes are all padding rows has nothing to drain
  if (rb0 + quad * 32 >= M) return nrm;
  const int row = rb0 + quad * 32 + lane;
  // the lower rows of a stacked product: their own epilogue and outputs
  const bool live = row < M, upper = !STACK || row < N;
  const int epi = upper ? EPI : EPI2;
  const int rowL = upper ? row : row - N;
  const int ox = upper ? (op >> 8) & 15 : (op >> 20) & 15;
  const int er = live ? s.rows(upper ? op & 15 : (op >> 16) & 15, N)[rowL] : 0;
  const int* const eY = s.cols((op >> 4) & 15, N);
  double2* const o0b = W + ox * NN + rowL;
  double2* const o1b = W + (upper ? (op >> 12) & 15 : (op >> 24) & 15) * NN + rowL;   // aux
  // column exponents of the outputs (a warp's rows may belong to both products)
  const int oU = (op >> 8) & 15, oL = (op >> 20) & 15;
  // (matrices 6 and 7, M1 and M2, are left factors only)
  int* const cU = (last && oU >= 3 && oU != 6 && oU != 7 && (!STACK || rb0 + quad * 32 < N)) ? s.cols(oU, N) : nullptr;
  int* const cL = (last && STACK && oL >= 3 && oL != 6 && oL != 7 && rb0 + quad * 32 + 31 >= N) ? s.cols(oL, N) : nullptr;
  unsigned rmax = 0;                       // upper words without sign: ordered like exponents
  const uint32_t tq = s.t().tslot + ((uint32_t)(quad * 32) << 16);
  // two columns at a time: the four warps of a quadrant share any pass width evenly (in
  // fours, 24 and 40 columns took two and three rounds of four instead of 1.5 and 2.5:
  // a product at Ndim 40 took 33.8 k cycles instead of 32.4)
#pragma unroll 1
  for (int c0 = hw * 2; c0 < width; c0 += 8) {
    uint32_t v[2][NACC][2];
    uint32_t ta = tq + (uint32_t)c0;
#pragma unroll
    for (int a = 0; a < NACC; ++a)
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        tmem_ld2(ta, v[comp][a]);
        ta += (uint32_t)width;
      }
    const int j0 = jb + c0;
    const bool on0 = live && j0 < N, on1 = live && j0 + 1 < N;
    double2* const p0 = o0b + (size_t)j0 * N;
    double2* const q0 = o1b + (size_t)j0 * N;
    double2 old0[2], old1[2];                 // the epilogue's loads
    old0[0] = old0[1] = old1[0] = old1[1] = make_double2(0.0, 0.0);
    if (epi == OZ_ADD2 || epi == OZ_ADDTO) {
      if (on0) old1[0] = q0[0];
      if (on1) old1[1] = q0[N];
    }
    if (epi == OZ_ADD2 || !first) {
      if (on0) old0[0] = p0[0];
      if (on1) old0[1] = p0[N];
    }
    tmem_wait_ld();
    double2 val[2];
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {          // without branches: four values in flight
      const int ee = er + eY[min(j0 + jj, N - 1)];
      uint32_t ar[NACC], ai[NACC];
#pragma unroll
      for (int a = 0; a < NACC; ++a) {
        ar[a] = v[0][a][jj];
        ai[a] = v[1][a][jj];
      }
      val[jj] = make_double2(K::value(ar, ee), K::value(ai, ee));
    }
    if (K::POISON) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
        if (max(er, eY[min(j0 + jj, N - 1)]) == 2047) {
          val[jj].x = __longlong_as_double(0x7FF8000000000000LL);
          val[jj].y = val[jj].x;
        }
    }
    if (epi == OZ_ADD2) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        old1[jj].x += val[jj].x;
        old1[jj].y += val[jj].y;
        val[jj].x += old0[jj].x;
        val[jj].y += old0[jj].y;
      }
      if (on0) q0[0] = old1[0];
      if (on1) q0[N] = old1[1];
    } else if (epi == OZ_IMINUS) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        if (first) {
          val[jj] = make_double2(-val[jj].x, -val[jj].y);
          // (one of the warp's rows is on the diagonal; FP64 adds are not free: two a clock)
          if ((unsigned)(j0 + jj - rb0 - quad * 32) < 32u && rowL == j0 + jj)
            val[jj].x = dsub_here(val[jj].x, -1.0);
        } else {
          val[jj] = make_double2(dsub_here(old0[jj].x, val[jj].x), dsub_here(old0[jj].y, val[jj].y));
        }
      }
    } else if (epi == OZ_ADDTO || !first) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const double2 o = first ? old1[jj] : old0[jj];
        val[jj].x += o.x;
        val[jj].y += o.y;
      }
    }
    if (on0) p0[0] = val[0];
    if (on1) p0[N] = val[1];
    if (last && (epi == OZ_STORE_NORM || epi == OZ_IMINUS)) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        if (!(jj ? on1 : on0)) continue;
        const float fr = upper_f32(val[jj].x), fi = upper_f32(val[jj].y);
        if (K::FRO && epi == OZ_IMINUS) nrm = fmaf(fr, fr, fmaf(fi, fi, nrm));
        else nrm += fr + fi;
      }
    }
    unsigned e[2];
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      e[jj] = max((unsigned)__double2hiint(val[jj].x) & 0x7FFFFFFFu,
                  (unsigned)__double2hiint(val[jj].y) & 0x7FFFFFFFu);
      if (!(jj ? on1 : on0)) e[jj] = 0;
      rmax = max(rmax, e[jj]);
    }
    if (cU) {
      const unsigned m0 = __reduce_max_sync(0xffffffffu, upper ? e[0] : 0u);
      const unsigned m1 = __reduce_max_sync(0xffffffffu, upper ? e[1] : 0u);
      if (lane < 2 && j0 + lane < N) atomicMax(&cU[j0 + lane], (int)((lane ? m1 : m0) >> 20));
    }
    if (cL) {
      const unsigned m0 = __reduce_max_sync(0xffffffffu, upper ? 0u : e[0]);
      const unsigned m1 = __reduce_max_sync(0xffffffffu, upper ? 0u : e[1]);
      if (lane < 2 && j0 + lane < N) atomicMax(&cL[j0 + lane], (int)((lane ? m1 : m0) >> 20));
    }
  }
  if (last && ox >= 3 && live) atomicMax(&s.rows(ox, N)[rowL], (int)(rmax >> 20));
  return nrm;
}

// C = X * Y through the epilogue EPI; with EPI2 >= 0, rows N .. 2N-1 of the
// tiles are a second product lo.X * Y with its own epilogue EPI2 and outputs
// (the first product's last, partly filled tile takes its first rows; each
// output element sees the same digits and sums as in a product of its own).
// Returns this thread's FP32 partial of a sum over the outputs: OZ_STORE_NORM
// and OZ_IMINUS sum |re| + |im| (OZ_IMINUS of a kind with FRO: re^2 + im^2).
template <class K>
__device__ __noinline__ float split_gemm(double2* __restrict__ const W, const uint32_t op,
                                         const int EPI, const int EPI2, const int N, const int NP,
                                         const int w0, const MxShared s) {
  SplitTail& sh = s.t();
  const int tid = threadIdx.x, warp = tid >> 5;
  const int M = EPI2 >= 0 ? 2 * N : N;           // rows of the tiles that hold outputs
  const int kper = k_part<K>(N);
  const int oU = (op >> 8) & 15, oL = (op >> 20) & 15;
  float nrm = 0.f;
  // the outputs' exponents start at the floor
  if (oU >= 3)
    for (int i = tid; i < 2 * N; i += SP_T) s.rows(oU, N)[i] = EXP_MIN;
  if (EPI2 >= 0 && oL >= 3)
    for (int i = tid; i < 2 * N; i += SP_T) s.rows(oL, N)[i] = EXP_MIN;
  __syncthreads();
  int abort = sh.abort;
  uint32_t c0 = sh.chunk;                        // first chunk of the tile
  int ahead = 0;                                 // chunks of the tile generated already
  Tile T = first_tile(N, NP, w0, kper);
  for (bool more = true; more && !abort;) {
    const Tile C = T;                            // the current tile; T: the next one
    const int nch = C.chunks();
    more = next_tile(T, M, N, NP, w0, kper);
    if (warp == 0) {
      // one thread issues the tile's MMAs as its chunks become complete
      int ab = 0;
      if (elect_one()) {
        const int slot = K::SLOT + (C.width == w0 ? 0 : 1);
        const IssueTab* const tab = sh.tabs + slot;
        const int n = sh.ntab[slot];
        const uint32_t tmem = sh.tslot;
        for (int c = 0; c < nch; ++c) {
          const uint32_t q = c0 + c;
          if (!mbar_wait(&sh.full[q & 1], (q >> 1) & 1, sh.spin)) {
            ab = 1;
            break;
          }
          tc_fence_after();
          split_issue<K>(tab, n, saddr(s.base()) + (q & 1) * s.stage, tmem, C.width, c > 0);
          mma_commit(&sh.empty[q & 1]);
          sh.issued = q + 1;
        }
      }
      __syncwarp();
      abort |= __any_sync(0xffffffffu, ab);
    } else {
      // this tile's chunks and the first two of the next one
      if (ahead < nch) abort |= split_generate<K>(W, op, N, M, C, ahead, nch, c0 + ahead, s);
      if (more && !abort) {
        ahead = min(2, T.chunks());
        abort |= split_generate<K>(W, op, N, M, T, 0, ahead, c0 + nch, s);
      }
    }
    // all MMAs of this tile: the last commit covers every earlier one
    const uint32_t ql = c0 + nch - 1;
    c0 += nch;
    if (!abort && !mbar_wait(&sh.empty[ql & 1], (ql >> 1) & 1, sh.spin)) abort = 1;
    __syncwarp();
    if (!__any_sync(0xffffffffu, abort)) {
      tc_fence_after();
      nrm = split_drain<K>(W, op, EPI, EPI2, N, M, C, nrm, s);
    }
    tc_fence_before();
    abort = __syncthreads_or(abort);
    tc_fence_after();
  }
  if (tid == 0) {
    sh.chunk = c0;
    sh.abort = abort;
  }
  __syncthreads();
  return nrm;
}

__device__ float block_sum_f(float v, const MxShared s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if (lane == 0) s.t().red[warp] = v;
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x == 0) {
    for (int w = 0; w < nw; ++w) t += s.t().red[w];
    s.t().red[0] = t;
  }
  __syncthreads();
  t = s.t().red[0];
  __syncthreads();
  return t;
}

// block sum in FP64 (16 warps: the 32-float reduction area holds 16 doubles)
static_assert(SP_T / 32 <= 16, "block_sum_d keeps one double per warp in s.red");
__device__ double block_sum_d(double v, const MxShared s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* red = reinterpret_cast<double*>(s.t().red);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < nw; ++w) t += red[w];
    red[0] = t;
  }
  __syncthreads();
  t = red[0];
  __syncthreads();
  return t;
}

// The convergence test sum_ij |alpha_ij| <= tol (src/surfgreen.f90:120-122).
// The product that made alpha summed u = sum (|re| + |im|) in FP32, which
// bounds the norm within u / sqrt(2) .. u; only where these bounds (with the
// FP32 sum's own error) do not decide is the FP64 sum taken, so 12.5 k FP64
// square roots an iteration (at Ndim 112, two FP64 operations a clock) are
// left out.  All threads.
__device__ bool converged(float part, const double2* __restrict__ Al, int N, double tol,
                          const MxShared s) {
  const double u = (double)block_sum_f(part, s);
  const int NN = N * N;
  if (u * (1.0 + 1e-4) + (double)NN * 3e-38 <= tol) return true;
  if (u * 0.7071 * (1.0 - 1e-4) > tol) return false;
  double d = 0.0;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) d += cabs64(Al[e].x, Al[e].y);
  return block_sum_d(d, s) <= tol;
}

// a complex float as one 64-bit register pair, for the packed FMA (two IEEE
// FP32 FMAs in one instruction)
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Gauss-Jordan without physical row swaps: row i of the working matrix stays
// in place and pos_of[i] / row_at[q] record the position it would hold in the
// swapped form.  Step t's pivot is the first maximal |re| + |im| of column t
// over the rows at positions >= t (izamax's rule in position order), so the
// pivots, and every FMA of every entry, are those of the swapped form; only
// the storage order differs.  For column t in registers (lane l of the warp
// holds rows l + 32 m): publishes the multiplier column (column t as it stands)
// to cb, the pivot's row to prow[t] and its reciprocal to *rslot, and moves the
// pivot to position t.
// Every lane prepares the reciprocal of its own best candidate while the warp
// finds the maximum (redux.sync of the key, then of the position), and the
// winning lane writes: the chain from the column to the published pivot has no
// division and no shuffle.
template <int R>
__device__ __forceinline__ void gj_pivot_publish(const unsigned long long (&x)[R], int t, int N,
                                                 float2* cb, float2* rslot, int* prow, int* singular,
                                                 int* pos_of, int* row_at) {
  const int lane = threadIdx.x & 31;
  const int rk = row_at[t];              // moves to the pivot's position
  int ps[R];
#pragma unroll
  for (int m = 0; m < R; ++m) ps[m] = pos_of[min(lane + 32 * m, N - 1)];
  unsigned bkey = 0;                      // key + 1; 0: no candidate
  int bpos = t, bm = 0;                   // (a valid position where a key wraps to none)
  float2 bv = make_float2(0.f, 0.f);
#pragma unroll
  for (int m = 0; m < R; ++m) {
    const int i = lane + 32 * m;
    const float2 v = unpack2(x[m]);
    if (i < N) cb[i] = v;
    const unsigned key = (i < N && ps[m] >= t)
                             ? (unsigned)__float_as_int(fabsf(v.x) + fabsf(v.y)) + 1u : 0u;
    if (key > bkey || (key == bkey && key && ps[m] < bpos)) {
      bkey = key;
      bpos = ps[m];
      bm = m;
      bv = v;
    }
  }
  const float inv_d = 1.0f / __fmaf_rn(bv.x, bv.x, __fmul_rn(bv.y, bv.y));
  const float2 rc = make_float2(bv.x * inv_d, -bv.y * inv_d);
  const unsigned kmax = __reduce_max_sync(0xffffffffu, bkey);
  const bool cand = bkey == kmax;
  const unsigned pmin = __reduce_min_sync(0xffffffffu, cand ? (unsigned)bpos : 0xffffffffu);
  if (cand && (unsigned)bpos == pmin) {   // one lane: positions are distinct
    const int brow = lane + 32 * bm;
    prow[t] = kmax == 1u ? -1 : brow;
    row_at[bpos] = rk;
    pos_of[rk] = bpos;
    row_at[t] = brow;
    pos_of[brow] = t;
    if (kmax == 1u) *singular = 1;
    else *rslot = rc;
  }
}

// One Gauss-Jordan step (pivot row p, reciprocal r, multiplier column cm in
// shared memory) applied to C columns held in registers (R rows a lane, packed),
// rows in place; column `own` (if any) is the pivot column itself.  Per entry
// v - f nk with the operations of four FMAs, re: -f.x nk.x, + f.y nk.y; im:
// -f.x nk.y, - f.y nk.x, as two packed ones.  The multipliers of a step are
// loaded once for all C columns.
template <int R, int C, int PM>
__device__ __forceinline__ void gj_step_at(unsigned long long (&x)[C][R],
                                           const unsigned long long (&fa)[R],
                                           const unsigned long long (&fb)[R], int pl, float2 r,
                                           int own) {
  const bool here = (threadIdx.x & 31) == pl;
  float2 nk[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const float2 v = unpack2(x[c][PM]);
    const float2 a = make_float2(__shfl_sync(0xffffffffu, v.x, pl), __shfl_sync(0xffffffffu, v.y, pl));
    nk[c] = make_float2(fmaf(a.x, r.x, -a.y * r.y), fmaf(a.x, r.y, a.y * r.x));
    if (C == 1 && c == own) {             // the pivot column becomes a column of the inverse
      nk[c] = r;
#pragma unroll
      for (int m = 0; m < R; ++m) x[c][m] = 0ull;
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const unsigned long long n0 = pack2(nk[c].x, nk[c].y), n1 = pack2(nk[c].y, nk[c].x);
#pragma unroll
    for (int m = 0; m < R; ++m) x[c][m] = fma2(fb[m], n1, fma2(fa[m], n0, x[c][m]));
    if (here) x[c][PM] = n0;
  }
}
// the row slot p / 32 of the pivot is the same for the whole warp: one branch
// instead of R selects a column
template <int R, int C>
__device__ __forceinline__ void gj_step_cols(unsigned long long (&x)[C][R],
                                             const float2* __restrict__ cm, int N, int p, float2 r,
                                             int own) {
  const int lane = threadIdx.x & 31;
  unsigned long long fa[R], fb[R];
#pragma unroll
  for (int m = 0; m < R; ++m) {
    const float2 f = cm[min(lane + 32 * m, N - 1)];      // rows >= N hold nothing
    fa[m] = pack2(-f.x, -f.x);
    fb[m] = pack2(f.y, -f.y);
  }
  const int pm = p >> 5, pl = p & 31;
#define WTG_GJ_AT(M)                                                                   \
  if constexpr (R > M) {                                                               \
    if (pm == M) gj_step_at<R, C, (M < R ? M : 0)>(x, fa, fb, pl, r, own);             \
  }
  WTG_GJ_AT(0) WTG_GJ_AT(1) WTG_GJ_AT(2) WTG_GJ_AT(3) WTG_GJ_AT(4)
  WTG_GJ_AT(5) WTG_GJ_AT(6) WTG_GJ_AT(7) WTG_GJ_AT(8) WTG_GJ_AT(9)
#undef WTG_GJ_AT
}

// barrier of the panel's warps (0 .. GJS_PANEL-1)
__device__ __forceinline__ void gj_panel_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(32 * GJS_PANEL) : "memory");
}

// M = w I - X (FP64, kept in Mi for the refinement, with its row exponents),
// then FP32 Gauss-Jordan with partial pivoting into G (FP64, with its row and
// column exponents).  Returns 1 on an exact zero pivot (G = identity then).
// Ndim <= 112, the matrix in shared memory.  The pivot steps run in panels of
// GJS_PANEL columns, one panel ahead of the rest: warps 0 .. GJS_PANEL-1 hold the
// next panel's columns in registers (lane l holds rows l, l + 32, ...), put them
// through the current panel's steps and factor them, one named barrier a step, the
// owner of the next column finding the next pivot and publishing its multiplier
// column; meanwhile the other warps read every remaining column once, up to C at a
// time, and put it through the current panel's steps.  Rows stay in place
// (gj_pivot_publish); the output reads them back in pivot order.
// What bounds it: the latency of the pivot steps (search, publication, barrier;
// about 1.4 k cycles each).  Alone on the chip an inverse takes 147.8 us at Ndim
// 112 and 32.9 at 40; with panels of 16 by all warps and the rest after each panel
// 172.5 and 37.9; panels of 4 175.2 and 35.1; panels factored by one warp in
// registers 232 and 37.0.  Same operations per entry, in the same order, in all.
template <int R>
__device__ __noinline__ int gj32_start(const double2* __restrict__ X, double2 w, int N,
                                       double2* __restrict__ const W, int iM, int iG,
                                       const MxShared s) {
  constexpr int C = R == 2 ? 3 : 6;       // trailing columns a warp holds at a time
  const size_t NN = (size_t)N * N;
  double2* __restrict__ const Mi = W + iM * NN;
  double2* __restrict__ const G = W + iG * NN;
  SplitTail& sh = s.t();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int nwarp = SP_T / 32;
  float2* __restrict__ sM = reinterpret_cast<float2*>(s.base());
  float2* __restrict__ Cm = sM + (size_t)N * N;          // [2][GJS_PANEL][N] multiplier columns
  float2* __restrict__ recip = sh.recip;                 // [2][GJS_PANEL]
  int* __restrict__ prow = sh.prow;                      // pivot rows
  int* __restrict__ misc = sh.misc;
  int* __restrict__ pos_of = sh.pos_of;
  int* __restrict__ row_at = sh.row_at;
  int rmax[R];
#pragma unroll
  for (int q = 0; q < R; ++q) rmax[q] = 0;
#pragma unroll 2
  for (int j = warp; j < N; j += nwarp) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = lane + 32 * q;
      if (i < N) {
        const size_t e = (size_t)i + (size_t)j * N;
        const double2 x = X[e];
        double2 m = make_double2(-x.x, -x.y);
        if (i == j) m = make_double2(w.x - x.x, w.y - x.y);
        Mi[e] = m;
        sM[e] = make_float2(d2f_bits(m.x), d2f_bits(m.y));
        rmax[q] = max(rmax[q], max(bexp(m.x), bexp(m.y)));
      }
    }
  }
  int* const eM = s.rows(iM, N);
  int* const eGr = s.rows(iG, N);
  int* const eGc = s.cols(iG, N);
  for (int i = tid; i < N; i += SP_T) {
    pos_of[i] = i;
    row_at[i] = i;
    eM[i] = EXP_MIN;
    eGr[i] = EXP_MIN;
  }
  if (tid < 2) misc[2 + tid] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (lane + 32 * q < N) atomicMax(&eM[lane + 32 * q], rmax[q]);
  // warps 0 .. GJS_PANEL-1, a column each: the panel at k0 (pb columns) through the
  // pbb steps of the panel before it, factored into buffer b, and written back
  auto panel = [&](int k0, int pb, int pbb, int b) {
    float2* const cm = Cm + b * GJS_PANEL * N;
    const float2* const cb = Cm + (b ^ 1) * GJS_PANEL * N;
    float2* const rc = recip + b * GJS_PANEL;
    float2* const col = sM + (size_t)(k0 + warp) * N;
    unsigned long long xp[1][R];
#pragma unroll
    for (int m = 0; m < R; ++m) {
      const int i = lane + 32 * m;
      const float2 v = (warp < pb && i < N) ? col[i] : make_float2(0.f, 0.f);
      xp[0][m] = pack2(v.x, v.y);
    }
    if (warp < pb)
      for (int t = 0; t < pbb; ++t)
        gj_step_cols<R, 1>(xp, cb + t * N, N, prow[k0 - pbb + t], recip[(b ^ 1) * GJS_PANEL + t], -1);
    auto publish = [&](int t) {
      gj_pivot_publish<R>(xp[0], k0 + t, N, cm + t * N, rc + t, prow, misc + 2 + b, pos_of, row_at);
    };
    if (warp == 0) publish(0);
    gj_panel_sync();
    for (int t = 0; t < pb; ++t) {
      const int p = prow[k0 + t];
      if (p < 0) break;
      if (warp < pb) {
        gj_step_cols<R, 1>(xp, cm + t * N, N, p, rc[t], warp == t ? 0 : -1);
        if (warp == t + 1) publish(t + 1);
      }
      gj_panel_sync();
    }
    if (warp < pb) {
#pragma unroll
      for (int m = 0; m < R; ++m) {
        const int i = lane + 32 * m;
        if (i < N) col[i] = unpack2(xp[0][m]);
      }
    }
  };
  if (warp < GJS_PANEL) panel(0, min(GJS_PANEL, N), 0, 0);
  __syncthreads();
  for (int k0 = 0, b = 0; k0 < N && !misc[2 + b]; k0 += GJS_PANEL, b ^= 1) {
    const int pb = min(GJS_PANEL, N - k0), pn = min(GJS_PANEL, N - k0 - pb);
    if (pn > 0 && warp < GJS_PANEL) {
      panel(k0 + pb, pn, pb, b ^ 1);
    } else {
      // the columns outside the two panels (after the last one every warp's), C at a time
      const int first = pn > 0 ? GJS_PANEL : 0, step = nwarp - first, skip = pb + pn;
      const float2* const cm = Cm + b * GJS_PANEL * N;
      for (int o0 = warp - first; o0 < N - skip; o0 += C * step) {
        unsigned long long x[C][R];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = o0 + c * step;
          const float2* col = sM + (size_t)(o < k0 ? o : o + skip) * N;
#pragma unroll
          for (int m = 0; m < R; ++m) {
            const int i = lane + 32 * m;
            const float2 v = (o < N - skip && i < N) ? col[i] : make_float2(0.f, 0.f);
            x[c][m] = pack2(v.x, v.y);
          }
        }
        for (int t = 0; t < pb; ++t)
          gj_step_cols<R, C>(x, cm + t * N, N, prow[k0 + t], recip[b * GJS_PANEL + t], -1);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = o0 + c * step;
          float2* col = sM + (size_t)(o < k0 ? o : o + skip) * N;
#pragma unroll
          for (int m = 0; m < R; ++m) {
            const int i = lane + 32 * m;
            if (o < N - skip && i < N) col[i] = unpack2(x[c][m]);
          }
        }
      }
    }
    __syncthreads();
  }
  const int singular = misc[2] | misc[3];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; ++q) rmax[q] = 0;
#pragma unroll 2
  for (int j = warp; j < N; j += nwarp) {
    const int cj = pos_of[j];             // the row swaps as column swaps of the inverse
    int cmax = EXP_MIN;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = lane + 32 * q;
      if (i < N) {
        double2 g = make_double2(i == j ? 1.0 : 0.0, 0.0);
        if (!singular) {
          const float2 v = sM[row_at[i] + (size_t)cj * N];
          g = make_double2(f2d_bits(v.x), f2d_bits(v.y));
        }
        G[(size_t)i + (size_t)j * N] = g;
        const int e = max(bexp(g.x), bexp(g.y));
        rmax[q] = max(rmax[q], e);
        cmax = max(cmax, e);
      }
    }
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if (lane == 0) eGc[j] = cmax;
  }
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (lane + 32 * q < N) atomicMax(&eGr[lane + 32 * q], rmax[q]);
  __syncthreads();
  return singular;
}

// As gj32_start for Ndim above the shared-memory limit: the FP32 matrix lives
// in global memory (Wf, N x N float2) and the pivot steps run in panels of
// MX_PANEL columns.  A panel's columns stay in registers (warp w owns panel
// column w, lane l rows l, l+32, ..., R rows per lane); each step updates them with
// one barrier, the owner of the next column publishing the next pivot and its
// multiplier column (look-ahead).  Then every other column is read once into
// registers, put through the panel's steps in order and written back.  Rows
// stay in place as in gj32_start.
template <int R>
__device__ __noinline__ int gj32_global(const double2* __restrict__ X, double2 w, int N,
                                        double2* __restrict__ const W, int iM, int iG, int iW,
                                        const MxShared s) {
  const size_t NN = (size_t)N * N;
  double2* __restrict__ const Mi = W + iM * NN;
  double2* __restrict__ const G = W + iG * NN;
  SplitTail& sh = s.t();
  constexpr int C = R <= 5 ? 3 : 2;       // columns a warp takes at a time
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int nwarp = SP_T / 32;
  float2* __restrict__ const Wf = reinterpret_cast<float2*>(W + iW * NN);
  // [MX_MAXN][MX_PANEL] multiplier columns of the panel
  float2* __restrict__ Cm = reinterpret_cast<float2*>(s.base());
  float2* __restrict__ recip = sh.recip;
  int* __restrict__ misc = sh.misc;
  int* const prow = sh.prow;                     // pivot rows of the steps
  int* __restrict__ pos_of = sh.pos_of;
  int* __restrict__ row_at = sh.row_at;
  int rmax[R];
#pragma unroll
  for (int q = 0; q < R; ++q) rmax[q] = 0;
  for (int j = warp; j < N; j += nwarp) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = lane + 32 * q;
      if (i < N) {
        const size_t e = (size_t)i + (size_t)j * N;
        const double2 x = X[e];
        double2 m = make_double2(-x.x, -x.y);
        if (i == j) m = make_double2(w.x - x.x, w.y - x.y);
        Mi[e] = m;
        Wf[e] = make_float2(d2f_bits(m.x), d2f_bits(m.y));
        rmax[q] = max(rmax[q], max(bexp(m.x), bexp(m.y)));
      }
    }
  }
  int* const eM = s.rows(iM, N);
  int* const eGr = s.rows(iG, N);
  int* const eGc = s.cols(iG, N);
  for (int i = tid; i < N; i += SP_T) {
    pos_of[i] = i;
    row_at[i] = i;
    eM[i] = EXP_MIN;
    eGr[i] = EXP_MIN;
  }
  if (tid == 0) misc[1] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (lane + 32 * q < N) atomicMax(&eM[lane + 32 * q], rmax[q]);
  for (int k0 = 0; k0 < N; k0 += MX_PANEL) {
    const int pb = min(MX_PANEL, N - k0);
    {
      unsigned long long xp[1][R];        // this warp's panel column
      float2* const col = Wf + (size_t)(k0 + warp) * N;
#pragma unroll
      for (int m = 0; m < R; ++m) {
        const int i = lane + 32 * m;
        const float2 v = (warp < pb && i < N) ? col[i] : make_float2(0.f, 0.f);
        xp[0][m] = pack2(v.x, v.y);
      }
      auto publish = [&](int t) {
        gj_pivot_publish<R>(xp[0], k0 + t, N, Cm + t * N, &recip[t], prow, misc + 1, pos_of, row_at);
      };
      if (warp == 0) publish(0);
      __syncthreads();
      for (int t = 0; t < pb; ++t) {
        const int p = prow[k0 + t];
        if (p < 0) break;
        if (warp < pb) {
          gj_step_cols<R, 1>(xp, Cm + t * N, N, p, recip[t], warp == t ? 0 : -1);
          if (warp == t + 1) publish(t + 1);
        }
        __syncthreads();
      }
      if (misc[1]) break;
      if (warp < pb) {                    // panel column back to memory
#pragma unroll
        for (int m = 0; m < R; ++m) {
          const int i = lane + 32 * m;
          if (i < N) col[i] = unpack2(xp[0][m]);
        }
      }
    }
    // every column outside the panel through the panel's steps, C at a time
    for (int o0 = warp; o0 < N - pb; o0 += C * nwarp) {
      const int nc = min(C, (N - pb - o0 + nwarp - 1) / nwarp);
      unsigned long long x[C][R];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int o = o0 + c * nwarp;
        const float2* col = Wf + (size_t)(o < k0 ? o : o + pb) * N;
#pragma unroll
        for (int m = 0; m < R; ++m) {
          const int i = lane + 32 * m;
          const float2 v = (c < nc && i < N) ? col[i] : make_float2(0.f, 0.f);
          x[c][m] = pack2(v.x, v.y);
        }
      }
      for (int t = 0; t < pb; ++t)
        gj_step_cols<R, C>(x, Cm + t * N, N, prow[k0 + t], recip[t], -1);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int o = o0 + c * nwarp;
        float2* col = Wf + (size_t)(o < k0 ? o : o + pb) * N;
#pragma unroll
        for (int m = 0; m < R; ++m) {
          const int i = lane + 32 * m;
          if (c < nc && i < N) col[i] = unpack2(x[c][m]);
        }
      }
    }
    __syncthreads();
  }
  const int singular = misc[1];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; ++q) rmax[q] = 0;
  for (int j = warp; j < N; j += nwarp) {
    const int cj = pos_of[j];             // the row swaps as column swaps of the inverse
    int cmax = EXP_MIN;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = lane + 32 * q;
      if (i < N) {
        double2 g = make_double2(i == j ? 1.0 : 0.0, 0.0);
        if (!singular) {
          const float2 v = Wf[row_at[i] + (size_t)cj * N];
          g = make_double2(f2d_bits(v.x), f2d_bits(v.y));
        }
        G[(size_t)i + (size_t)j * N] = g;
        const int e = max(bexp(g.x), bexp(g.y));
        rmax[q] = max(rmax[q], e);
        cmax = max(cmax, e);
      }
    }
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if (lane == 0) eGc[j] = cmax;
  }
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (lane + 32 * q < N) atomicMax(&eGr[lane + 32 * q], rmax[q]);
  __syncthreads();
  return singular;
}

// FP32 inverse of w I - X by Ndim: M to workspace matrix iM, the inverse to iG, iR as work
__device__ __forceinline__ int gj32(const double2* X, double2 w, int N, double2* W, int iM, int iG,
                                    int iR, const MxShared s) {
  return N <= 64              ? gj32_start<2>(X, w, N, W, iM, iG, s)
         : N <= MX_SMEM_GJ_N ? gj32_start<4>(X, w, N, W, iM, iG, s)
         : N <= 160        ? gj32_global<5>(X, w, N, W, iM, iG, iR, s)
         : N <= 224        ? gj32_global<7>(X, w, N, W, iM, iG, iR, s)
                           : gj32_global<MX_ROWS>(X, w, N, W, iM, iG, iR, s);
}

__device__ __forceinline__ void swap_mat(int& a, int& b) {
  const int t = a;
  a = b;
  b = t;
}

// exponents of b = a^dagger from a's
__device__ __forceinline__ void exps_dagger(int b, int a, int N, const MxShared s) {
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    s.rows(b, N)[i] = s.cols(a, N)[i];
    s.cols(b, N)[i] = s.rows(a, N)[i];
  }
  __syncthreads();
}

// issue tables of a plan's products (lanes of warp 0); visible to the issuing
// thread after the next barrier
template <class K7, class K4>
__device__ void split_tables(const MxPlan& pl, const MxShared s) {
  const MxPlan p4 = split_plan4(pl);
  const int t = threadIdx.x;
  if (t < 4) {
    const MxPlan& p = t < 2 ? pl : p4;
    const int last = p.NP - (p.ncb - 1) * p.w0;
    const int w = (t & 1) ? last : p.w0;
    if (t < 2) issue_table<K7>(s.t().tabs + t, s.t().ntab + t, w);
    else issue_table<K4>(s.t().tabs + t, s.t().ntab + t, w);
  }
}

// tensor-memory allocation and mbarriers of a CTA (all threads)
__device__ void mx_setup(const MxShared s, unsigned spin_limit) {
  const int tid = threadIdx.x;
  SplitTail& sh = s.t();
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(&sh.full[b])), "r"(SP_GEN / 32));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&sh.empty[b])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sh.chunk = 0;
    sh.issued = 0;
    sh.abort = 0;
    sh.spin = spin_limit;
  }
  if ((tid >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     saddr(&sh.tslot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

// every committed MMA must finish before tensor memory is released: this wait
// keeps the built-in bound whatever a test set for the pipeline's waits
__device__ void mx_teardown(const MxShared s) {
  SplitTail& sh = s.t();
  __syncthreads();
  if (threadIdx.x == 0 && sh.issued > 0) {
    const uint32_t q = sh.issued - 1;
    mbar_wait(&sh.empty[q & 1], (q >> 1) & 1, 0u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tslot), "r"(512));
}
