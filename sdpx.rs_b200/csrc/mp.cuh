// Correctly rounded MpFloat<N> arithmetic on the GPU (N 64-bit limbs, round to nearest, ties to
// even: the MPFR contract of crates/arithmetic/src/lib.rs that the reference's MpFloat follows).
//
// Element layout (the reference's in-memory MpFloat<N>, lib.rs:333-340): u64 limbs[N], least
// significant first, i32 kind = sign * MPFR kind (2 zero, 3 regular), i32 exponent; a regular
// value is M * 2^(exponent - 64N) with the top bit of M set.
//
// Everything is a template on N with every loop over words unrolled, so mantissas, products and
// accumulators live in registers (32-bit words, carries by add.cc / madc chains) instead of
// run-time-length loops over local memory: an exact product of two 256-bit mantissas is 64
// multiply-adds.  Every operation forms its exact result (or the exact result's leading words
// with a sticky bit) and rounds it once:
//   addsub              aligned sum with a 64-bit guard and a sticky bit (operands more than
//                       64N + 64 bits apart: the larger one unchanged)
//   mul                 2N-limb product
//   recip, divide,      the integer quotient floor(2^(128N + 2) / M), floor(M_a 2^(64N + 2) / M_b)
//   root                or root floor(sqrt(M 2^e)) with its remainder folded into a sticky bit;
//                       the quotient or root from a Newton estimate corrected exactly by its
//                       multiword remainder
//   dot<N, G>           a - sum x_c y_c (or sum x_c y_c) by G lanes, exact in a two's-complement
//                       fixed-point accumulator and rounded once (the exact dot of
//                       exactdot.rs:53-70).  Terms whose scales span at most kSpanBits accumulate in
//                       registers; up to kAccWords words in local memory; wider ones report failure.
// The arithmetic compiles for the host too (plain C++ in place of the carry chains), where the
// tests compare it with exact integers.
#pragma once
#include <climits>
#include <cmath>
#include <cstdint>
#include <type_traits>

#if defined(__CUDACC__)
#define MPD_FN __host__ __device__ __forceinline__
#define MPD_CALL __host__ __device__ __noinline__
#else
#define MPD_FN inline
#define MPD_CALL inline
#endif

namespace mpd {

constexpr int kMaxN = 8;        // limbs: up to 512-bit values
constexpr int kAccWords = 40;   // exact-dot accumulator: 2560 bits of spread + width
constexpr int kKindZero = 2, kKindRegular = 3;
constexpr int kExpMax = (1 << 30) - 1;

template <int N>
struct Val {
  uint32_t m[2 * N];  // mantissa, top bit set (unless zero), least significant word first
  long long s;        // scale: value = (-1)^neg M 2^s
  bool neg, zero;
};

// ---- word arithmetic ----

MPD_FN uint32_t funnel_l(uint32_t lo, uint32_t hi, int r) {  // high word of (hi:lo) << r, 0 <= r < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, r);
#else
  return r ? (hi << r) | (lo >> (32 - r)) : hi;
#endif
}
MPD_FN uint32_t funnel_r(uint32_t lo, uint32_t hi, int r) {  // low word of (hi:lo) >> r, 0 <= r < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, r);
#else
  return r ? (lo >> r) | (hi << (32 - r)) : lo;
#endif
}
MPD_FN int clz32(uint32_t v) {
#if defined(__CUDA_ARCH__)
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// a[0..K) += b[0..K) + c; the carry out.  (The asm blocks below write their outputs last: operands
// of equal value may share a register with an output.)
template <int K>
MPD_FN uint32_t add_words(uint32_t* a, const uint32_t* b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  constexpr int K4 = K / 4 * 4;
#pragma unroll
  for (int i = 0; i < K4; i += 4)
    asm("{\n\t.reg .u32 t0, t1, t2, t3;\n\t"
        "add.cc.u32 t0, %13, 0xffffffff;\n\t"
        "addc.cc.u32 t0, %5, %9;\n\t"
        "addc.cc.u32 t1, %6, %10;\n\t"
        "addc.cc.u32 t2, %7, %11;\n\t"
        "addc.cc.u32 t3, %8, %12;\n\t"
        "addc.u32 %4, 0, 0;\n\t"
        "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\tmov.u32 %2, t2;\n\tmov.u32 %3, t3;\n\t}"
        : "=r"(a[i]), "=r"(a[i + 1]), "=r"(a[i + 2]), "=r"(a[i + 3]), "=r"(c)
        : "r"(a[i]), "r"(a[i + 1]), "r"(a[i + 2]), "r"(a[i + 3]), "r"(b[i]), "r"(b[i + 1]), "r"(b[i + 2]),
          "r"(b[i + 3]), "r"(c));
#pragma unroll
  for (int i = K4; i < K; ++i)
    asm("{\n\t.reg .u32 t0;\n\t"
        "add.cc.u32 t0, %4, 0xffffffff;\n\t"
        "addc.cc.u32 t0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;\n\t"
        "mov.u32 %0, t0;\n\t}"
        : "=r"(a[i]), "=r"(c)
        : "r"(a[i]), "r"(b[i]), "r"(c));
#else
  for (int i = 0; i < K; ++i) {
    const uint64_t t = (uint64_t)a[i] + b[i] + c;
    a[i] = (uint32_t)t;
    c = (uint32_t)(t >> 32);
  }
#endif
  return c;
}
// a[0..K) -= b[0..K); the borrow out.
template <int K>
MPD_FN uint32_t sub_words(uint32_t* a, const uint32_t* b) {
  uint32_t t[K];
#pragma unroll
  for (int i = 0; i < K; ++i) t[i] = ~b[i];
  return 1u - add_words<K>(a, t, 1u);
}
// a[0..K) += x (one word); the carry out.
template <int K>
MPD_FN uint32_t add_word(uint32_t* a, uint32_t x) {
  uint32_t z[K];
#pragma unroll
  for (int i = 0; i < K; ++i) z[i] = 0u;
  z[0] = x;
  return add_words<K>(a, z, 0u);
}
// a[0..K) = -a.
template <int K>
MPD_FN void neg_words(uint32_t* a) {
  uint32_t z[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    a[i] = ~a[i];
    z[i] = 0u;
  }
  add_words<K>(a, z, 1u);
}
template <int K>
MPD_FN bool is_zero(const uint32_t* a) {
  uint32_t o = 0;
#pragma unroll
  for (int i = 0; i < K; ++i) o |= a[i];
  return o == 0;
}
// sign of a - b over K words
template <int K>
MPD_FN int cmp_words(const uint32_t* a, const uint32_t* b) {
  int r = 0;
#pragma unroll
  for (int i = 0; i < K; ++i) r = a[i] == b[i] ? r : (a[i] > b[i] ? 1 : -1);
  return r;
}

// One link of a multiply-accumulate chain: the P 64-bit words (acc[2i+1] : acc[2i]) += a[2i] * b,
// carry in and out in c.
template <int P>
MPD_FN void mac_link(uint32_t* acc, const uint32_t* a, uint32_t b, uint32_t& c) {
#if defined(__CUDA_ARCH__)
  if constexpr (P == 4) {
    asm("{\n\t.reg .u32 t0, t1, t2, t3, t4, t5, t6, t7;\n\t"
        "add.cc.u32 t0, %22, 0xffffffff;\n\t"
        "madc.lo.cc.u32 t0, %17, %21, %9;\n\t"
        "madc.hi.cc.u32 t1, %17, %21, %10;\n\t"
        "madc.lo.cc.u32 t2, %18, %21, %11;\n\t"
        "madc.hi.cc.u32 t3, %18, %21, %12;\n\t"
        "madc.lo.cc.u32 t4, %19, %21, %13;\n\t"
        "madc.hi.cc.u32 t5, %19, %21, %14;\n\t"
        "madc.lo.cc.u32 t6, %20, %21, %15;\n\t"
        "madc.hi.cc.u32 t7, %20, %21, %16;\n\t"
        "addc.u32 %8, 0, 0;\n\t"
        "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\tmov.u32 %2, t2;\n\tmov.u32 %3, t3;\n\t"
        "mov.u32 %4, t4;\n\tmov.u32 %5, t5;\n\tmov.u32 %6, t6;\n\tmov.u32 %7, t7;\n\t}"
        : "=r"(acc[0]), "=r"(acc[1]), "=r"(acc[2]), "=r"(acc[3]), "=r"(acc[4]), "=r"(acc[5]), "=r"(acc[6]),
          "=r"(acc[7]), "=r"(c)
        : "r"(acc[0]), "r"(acc[1]), "r"(acc[2]), "r"(acc[3]), "r"(acc[4]), "r"(acc[5]), "r"(acc[6]), "r"(acc[7]),
          "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b), "r"(c));
  } else if constexpr (P == 2) {
    asm("{\n\t.reg .u32 t0, t1, t2, t3;\n\t"
        "add.cc.u32 t0, %12, 0xffffffff;\n\t"
        "madc.lo.cc.u32 t0, %9, %11, %5;\n\t"
        "madc.hi.cc.u32 t1, %9, %11, %6;\n\t"
        "madc.lo.cc.u32 t2, %10, %11, %7;\n\t"
        "madc.hi.cc.u32 t3, %10, %11, %8;\n\t"
        "addc.u32 %4, 0, 0;\n\t"
        "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\tmov.u32 %2, t2;\n\tmov.u32 %3, t3;\n\t}"
        : "=r"(acc[0]), "=r"(acc[1]), "=r"(acc[2]), "=r"(acc[3]), "=r"(c)
        : "r"(acc[0]), "r"(acc[1]), "r"(acc[2]), "r"(acc[3]), "r"(a[0]), "r"(a[2]), "r"(b), "r"(c));
  } else {
    asm("{\n\t.reg .u32 t0, t1;\n\t"
        "add.cc.u32 t0, %7, 0xffffffff;\n\t"
        "madc.lo.cc.u32 t0, %5, %6, %3;\n\t"
        "madc.hi.cc.u32 t1, %5, %6, %4;\n\t"
        "addc.u32 %2, 0, 0;\n\t"
        "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\t}"
        : "=r"(acc[0]), "=r"(acc[1]), "=r"(c)
        : "r"(acc[0]), "r"(acc[1]), "r"(a[0]), "r"(b), "r"(c));
  }
#else
  for (int i = 0; i < P; ++i) {
    const unsigned __int128 t = (unsigned __int128)((uint64_t)a[2 * i] * b) +
                                (((uint64_t)acc[2 * i + 1] << 32) | acc[2 * i]) + c;
    acc[2 * i] = (uint32_t)t;
    acc[2 * i + 1] = (uint32_t)(t >> 32);
    c = (uint32_t)(t >> 64);
  }
#endif
}
// The 2N words at acc += sum_i a[2i] b 2^(64 i); the carry out.
template <int N>
MPD_FN uint32_t mac_chain(uint32_t* acc, const uint32_t* a, uint32_t b) {
  uint32_t c = 0;
  constexpr int N4 = N / 4 * 4;
#pragma unroll
  for (int i = 0; i < N4; i += 4) mac_link<4>(acc + 2 * i, a + 2 * i, b, c);
  if constexpr ((N & 3) >= 2) mac_link<2>(acc + 2 * N4, a + 2 * N4, b, c);
  if constexpr (N & 1) mac_link<1>(acc + 2 * (N - 1), a + 2 * (N - 1), b, c);
  return c;
}

// P (4N words) = a * b (2N words each).  The products a_i b_j with i + j even and with i + j odd
// are summed in two accumulators (the second one word up), so that every chain adds aligned
// 64-bit products with one running carry.
template <int N>
MPD_FN void mul_words(uint32_t* P, const uint32_t* a, const uint32_t* b) {
  constexpr int W = 2 * N;
  uint32_t O[2 * W];
#pragma unroll
  for (int i = 0; i < W; i += 2) {
    const uint64_t e = (uint64_t)a[i] * b[0], o = (uint64_t)a[i + 1] * b[0];
    P[i] = (uint32_t)e;
    P[i + 1] = (uint32_t)(e >> 32);
    O[i] = (uint32_t)o;
    O[i + 1] = (uint32_t)(o >> 32);
  }
#pragma unroll
  for (int i = W; i < 2 * W; ++i) P[i] = O[i] = 0u;
#pragma unroll
  for (int j = 1; j < W; ++j) {
    if (j & 1) {
      const uint32_t c = mac_chain<N>(P + j + 1, a + 1, b[j]);
      if (j + 1 + W < 2 * W) P[j + 1 + W] += c;
      O[j - 1 + W] += mac_chain<N>(O + j - 1, a, b[j]);
    } else {
      P[j + W] += mac_chain<N>(P + j, a, b[j]);
      O[j + W] += mac_chain<N>(O + j, a + 1, b[j]);
    }
  }
  add_words<2 * W - 1>(P + 1, O, 0u);
}

// ---- rounding ----

template <int N>
MPD_FN Val<N> zero_val() {
  Val<N> v;
#pragma unroll
  for (int q = 0; q < 2 * N; ++q) v.m[q] = 0u;
  v.s = 0;
  v.neg = false;
  v.zero = true;
  return v;
}
template <int N>
MPD_FN Val<N> one_val() {
  Val<N> v = zero_val<N>();
  v.zero = false;
  v.m[2 * N - 1] = 1u << 31;
  v.s = 1 - 64LL * N;
  return v;
}

template <int K, int W>
struct ShiftStage {  // shift S left by W words while its top W words are zero, then by W/2, ...
  static MPD_FN void run(uint32_t* S, int& sh) {
    if (W < K) {
      uint32_t o = 0;
#pragma unroll
      for (int i = 0; i < W && i < K; ++i) o |= S[K - 1 - i];
      if (o == 0) {
#pragma unroll
        for (int i = K - 1; i >= 0; --i) S[i] = i >= W ? S[i >= W ? i - W : 0] : 0u;
        sh += 32 * W;
      }
    }
    ShiftStage<K, W / 2>::run(S, sh);
  }
};
template <int K>
struct ShiftStage<K, 0> {
  static MPD_FN void run(uint32_t*, int&) {}
};

// Shift the nonzero S (K <= 128 words) left until its top bit is set; the bits shifted.
template <int K>
MPD_FN int normalize(uint32_t* S) {
  int sh = 0;
  if (S[K - 1] == 0) ShiftStage<K, (K > 64 ? 64 : 32)>::run(S, sh);
  const int c = clz32(S[K - 1]) & 31;
#pragma unroll
  for (int i = K - 1; i > 0; --i) S[i] = funnel_l(S[i - 1], S[i], c);
  S[0] <<= c;
  return sh + c;
}

// S (K > 2N words, top bit set) * 2^scale rounded to N limbs, ties to even.
template <int N, int K>
MPD_FN Val<N> round_top(const uint32_t* S, bool neg, long long scale) {
  Val<N> v;
  v.zero = false;
  v.neg = neg;
#pragma unroll
  for (int q = 0; q < 2 * N; ++q) v.m[q] = S[K - 2 * N + q];
  uint32_t sticky = S[K - 2 * N - 1] << 1;
#pragma unroll
  for (int i = 0; i < K - 2 * N - 1; ++i) sticky |= S[i];
  long long s = scale + 32 * (K - 2 * N);
  if ((S[K - 2 * N - 1] >> 31) && (sticky || (v.m[0] & 1u))) {
    if (add_word<2 * N>(v.m, 1u)) {  // carried out: the mantissa wrapped to zero
      v.m[2 * N - 1] = 1u << 31;
      s += 1;
    }
  }
  v.s = s;
  return v;
}

// ---- elements ----

template <int N>
MPD_FN Val<N> load(const unsigned char* p) {
  Val<N> v;
  const unsigned long long* l = reinterpret_cast<const unsigned long long*>(p);
  unsigned long long w[N + 1];
#pragma unroll
  for (int q = 0; q <= N; ++q) w[q] = l[q];
  const int kind = (int)(uint32_t)w[N], ex = (int)(uint32_t)(w[N] >> 32);
  v.zero = (kind == kKindZero || kind == -kKindZero);
  v.neg = kind < 0;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    v.m[2 * q] = v.zero ? 0u : (uint32_t)w[q];
    v.m[2 * q + 1] = v.zero ? 0u : (uint32_t)(w[q] >> 32);
  }
  v.s = (long long)ex - 64LL * N;
  return v;
}

// The scale and kind of an element alone: false for a zero.
template <int N>
MPD_FN bool load_scale(const unsigned char* p, long long* s) {
  const unsigned long long w = reinterpret_cast<const unsigned long long*>(p)[N];
  const int kind = (int)(uint32_t)w;
  *s = (long long)(int)(uint32_t)(w >> 32) - 64LL * N;
  return kind != kKindZero && kind != -kKindZero;
}

// Store v (zeros as +0); an exponent outside the MPFR range sets bit 4 (non-finite) of *status.
template <int N>
MPD_FN void store(unsigned char* p, const Val<N>& v, uint32_t* status) {
  unsigned long long* l = reinterpret_cast<unsigned long long*>(p);
  const long long ex = v.s + 64LL * N;
  const bool out = !v.zero && (ex > kExpMax || ex < -kExpMax);
#if defined(__CUDA_ARCH__)
  if (out && status) atomicOr(status, 4u);
#else
  if (out && status) *status |= 4u;
#endif
  const bool z = v.zero || out;
#pragma unroll
  for (int q = 0; q < N; ++q)
    l[q] = z ? 0ull : ((unsigned long long)v.m[2 * q + 1] << 32) | (unsigned long long)v.m[2 * q];
  const uint32_t kind = z ? (uint32_t)kKindZero : (uint32_t)(v.neg ? -kKindRegular : kKindRegular);
  l[N] = ((unsigned long long)(z ? 0u : (uint32_t)(int)ex) << 32) | kind;
}

// An intermediate for another thread of the CTA, 8N + 8 bytes: the value as it is in registers, its scale
// not held to the range of a stored element (the dot that an entry is reduced by may lie outside where
// the entry does not).
template <int N>
MPD_FN void stage(unsigned char* p, const Val<N>& v) {
  unsigned long long* l = reinterpret_cast<unsigned long long*>(p);
#pragma unroll
  for (int q = 0; q < N; ++q) l[q] = ((unsigned long long)v.m[2 * q + 1] << 32) | (unsigned long long)v.m[2 * q];
  l[N] = (unsigned long long)v.s << 2 | (v.neg ? 2u : 0u) | (v.zero ? 1u : 0u);
}
template <int N>
MPD_FN Val<N> unstage(const unsigned char* p) {
  Val<N> v;
  const unsigned long long* l = reinterpret_cast<const unsigned long long*>(p);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    v.m[2 * q] = (uint32_t)l[q];
    v.m[2 * q + 1] = (uint32_t)(l[q] >> 32);
  }
  v.s = (long long)l[N] >> 2;
  v.neg = l[N] & 2u;
  v.zero = l[N] & 1u;
  return v;
}

// ---- sums and products ----

// B >>= d bits over K words (d <= 32 K); bits shifted out are or-ed into the result's last bit.
template <int K, int W>
struct DropStage {
  static MPD_FN void run(uint32_t* B, int ws, uint32_t& lost) {
    if (ws & W) {
#pragma unroll
      for (int i = 0; i < W && i < K; ++i) lost |= B[i];
#pragma unroll
      for (int i = 0; i < K; ++i) B[i] = i + W < K ? B[i + W < K ? i + W : 0] : 0u;
    }
    DropStage<K, (2 * W <= K ? 2 * W : 0)>::run(B, ws, lost);
  }
};
template <int K>
struct DropStage<K, 0> {
  static MPD_FN void run(uint32_t*, int, uint32_t&) {}
};
template <int K>
MPD_FN void shift_right_sticky(uint32_t* B, int d) {
  uint32_t lost = 0;
  DropStage<K, 1>::run(B, d >> 5, lost);
  const int r = d & 31;
  lost |= B[0] & ((1u << r) - 1u);
#pragma unroll
  for (int i = 0; i < K - 1; ++i) B[i] = funnel_r(B[i], B[i + 1], r);
  B[K - 1] >>= r;
  B[0] |= lost ? 1u : 0u;
}

// a + sign * b, the exact sum rounded once (sign = -1: subtraction).  The smaller operand is
// aligned with 64 guard bits below the larger one's last bit and a sticky bit at the lowest of
// them: two operands within 64 bits of each other are summed exactly, and for the others the sum
// loses at most one leading bit, so the guard and the sticky bit decide the rounding.
template <int N>
MPD_CALL Val<N> addsub(Val<N> a, Val<N> b, int sign) {
  if (sign < 0) b.neg = !b.neg;
  if (b.zero) return a.zero ? zero_val<N>() : a;
  if (a.zero) return b;
  constexpr long long gap = 64LL * N + 64;
  const long long d = a.s - b.s;
  if (d > gap) return a;
  if (d < -gap) return b;
  constexpr int K = 2 * N + 2;
  const bool swap = d < 0;
  uint32_t A[K], B[K];
  A[0] = A[1] = B[0] = B[1] = 0u;
#pragma unroll
  for (int q = 0; q < 2 * N; ++q) {
    A[q + 2] = swap ? b.m[q] : a.m[q];
    B[q + 2] = swap ? a.m[q] : b.m[q];
  }
  long long s = (swap ? b.s : a.s) - 64;
  bool neg = swap ? b.neg : a.neg;
  shift_right_sticky<K>(B, (int)(swap ? -d : d));
  if (a.neg == b.neg) {
    if (add_words<K>(A, B, 0u)) {
      const uint32_t low = A[0] & 1u;
#pragma unroll
      for (int i = 0; i < K - 1; ++i) A[i] = funnel_r(A[i], A[i + 1], 1);
      A[K - 1] = (A[K - 1] >> 1) | (1u << 31);
      A[0] |= low;
      s += 1;
    }
  } else {
    if (sub_words<K>(A, B)) {  // equal scales, the second mantissa larger
      neg_words<K>(A);
      neg = !neg;
    }
    if (!(A[K - 1] >> 31)) {
      if (is_zero<K>(A)) return zero_val<N>();
      s -= normalize<K>(A);
    }
  }
  return round_top<N, K>(A, neg, s);
}

template <int N>
MPD_FN Val<N> mul(const Val<N>& a, const Val<N>& b) {
  if (a.zero || b.zero) return zero_val<N>();
  uint32_t P[4 * N];
  mul_words<N>(P, a.m, b.m);
  const int c = 1 - (int)(P[4 * N - 1] >> 31);  // the top bit is at most one place down
#pragma unroll
  for (int i = 4 * N - 1; i > 0; --i) P[i] = funnel_l(P[i - 1], P[i], c);
  P[0] <<= c;
  return round_top<N, 4 * N>(P, a.neg != b.neg, a.s + b.s - c);
}

// sign of a - b: -1, 0, 1.
template <int N>
MPD_FN int cmp(const Val<N>& a, const Val<N>& b) {
  if (a.zero && b.zero) return 0;
  if (a.zero) return b.neg ? 1 : -1;
  if (b.zero) return a.neg ? -1 : 1;
  if (a.neg != b.neg) return a.neg ? -1 : 1;
  int c = a.s != b.s ? (a.s > b.s ? 1 : -1) : cmp_words<2 * N>(a.m, b.m);
  return a.neg ? -c : c;
}

// ---- Newton estimates and the correctly rounded reciprocal, quotient and square root ----

// A value as (double in [0.5, 1), binary exponent): v = f 2^e, f its leading 53 bits.
template <int N>
MPD_FN double frac_exp(const Val<N>& v, long long* e) {
  const unsigned long long top = ((unsigned long long)v.m[2 * N - 1] << 32) | v.m[2 * N - 2];
  *e = v.s + 64LL * N;
  const double f = (double)(top >> 11) * 0x1p-53;
  return v.neg ? -f : f;
}

// f 2^e as a value (f a finite double).
template <int N>
MPD_FN Val<N> from_double(double f, long long e) {
  Val<N> v = zero_val<N>();
  if (f == 0.0) return v;
  int fe = 0;
  const double m = frexp(fabs(f), &fe);  // in [0.5, 1)
  const unsigned long long top = (unsigned long long)(m * 0x1p64);  // exact: 53 significant bits
  v.zero = false;
  v.neg = f < 0;
  v.m[2 * N - 1] = (uint32_t)(top >> 32);
  v.m[2 * N - 2] = (uint32_t)top;
  v.s = e + fe - 64LL * N;
  return v;
}

// 1 / x and 1 / sqrt(x) by Newton's iteration from an FP64 seed (quadratic convergence: four
// steps carry 53 bits past 512): accurate to a few units in the last place, not correctly
// rounded -- the Jacobi rotation parameters, whose orthogonality they bound, and the estimate
// that the correctly rounded root corrects.
template <int N>
MPD_CALL Val<N> recip_approx(Val<N> x) {
  long long e;
  const double f = frac_exp<N>(x, &e);
  Val<N> y = from_double<N>(1.0 / f, -e);
  const Val<N> two = from_double<N>(0.5, 2);
  constexpr int steps = N <= 2 ? 2 : (N <= 4 ? 3 : 4);
#pragma unroll 1
  for (int k = 0; k < steps; ++k) y = mul<N>(y, addsub<N>(two, mul<N>(x, y), -1));
  return y;
}
template <int N>
MPD_CALL Val<N> rsqrt_approx(Val<N> x) {  // x > 0
  long long e;
  const double f = frac_exp<N>(x, &e);
  // x = f 2^e: 1/sqrt(x) = (1/sqrt(f 2^(e mod 2))) 2^(-(e - e mod 2) / 2)
  const long long odd = e & 1;
  Val<N> y = from_double<N>(1.0 / sqrt(f * (odd ? 2.0 : 1.0)), -((e - odd) / 2));
  const Val<N> three = from_double<N>(0.75, 2);
  constexpr int steps = N <= 2 ? 2 : (N <= 4 ? 3 : 4);
#pragma unroll 1
  for (int k = 0; k < steps; ++k) {
    Val<N> t = addsub<N>(three, mul<N>(x, mul<N>(y, y)), -1);
    t.s -= 1;  // / 2
    y = mul<N>(y, t);
  }
  return y;
}

// Q (2N + 1 words) = floor(v 2^sh) for a positive v whose integer is at most 64N + 31 bits wide.
template <int N>
MPD_FN void to_words(const Val<N>& v, long long sh, uint32_t* Q) {
  const int t = (int)(v.s + sh) & 31;  // Q = M_v 2^t: the estimates below have 0 <= t < 32
  Q[2 * N] = funnel_l(v.m[2 * N - 1], 0u, t);
#pragma unroll
  for (int i = 2 * N - 1; i > 0; --i) Q[i] = funnel_l(v.m[i - 1], v.m[i], t);
  Q[0] = v.m[0] << t;
}

// R -= Q M modulo 2^(32 (2N + 2)), Q 2N + 1 words with a small top word, M 2N words: remainders of
// the estimates below stay within a few M, so their low 2N + 2 words are the whole remainder.
template <int N>
MPD_FN void sub_product(uint32_t* R, const uint32_t* Q, const uint32_t* M) {
  uint32_t P[4 * N];
  mul_words<N>(P, Q, M);
  uint32_t T[2 * N + 2];
#pragma unroll
  for (int i = 0; i < 2 * N + 2; ++i) T[i] = i < 4 * N ? P[i < 4 * N ? i : 0] : 0u;
  const uint64_t t0 = (uint64_t)Q[2 * N] * M[0];
  const uint32_t up[2] = {(uint32_t)t0, (uint32_t)(t0 >> 32) + Q[2 * N] * M[1]};
  add_words<2>(T + 2 * N, up, 0u);
  sub_words<2 * N + 2>(R, T);
}

// Q (2N + 1 words) = floor(R 2^(64N + 2) / M), for a positive R (2N + 1 words) below 2^(64N + 1) and not
// above 2 M, M (2N words) with its top bit set; returns whether the division leaves a remainder.
// Long division with signed digits: one of 2 bits (at most 8), then 2N of 32 bits, each the nearest
// integer to the leading three words of the remainder over the leading two of M in FP64 (off by less than
// 2^-18), so that |R| stays below 0.51 M.  A digit is one row of products and an FP64 estimate, about a
// hundred cycles at four limbs; Newton steps of full-width products took 7600 for the quotient.
template <int N>
MPD_FN bool long_division(uint32_t* R, const uint32_t* M, uint32_t* Q) {
  constexpr int W = 2 * N + 1;
  const double m = (double)M[2 * N - 1] * 0x1p32 + (double)M[2 * N - 2];
  const double y = 1.0 / m;
#pragma unroll
  for (int i = 0; i < W; ++i) Q[i] = 0u;
#pragma unroll 1
  for (int k = 0; k <= 2 * N; ++k) {
    const double r = (double)(int32_t)R[W - 1] * 0x1p64 + ((double)R[W - 2] * 0x1p32 + (double)R[W - 3]);
    const long long q = (long long)rint(r * (k == 0 ? 4.0 * y : 0x1p32 * y));
    const uint32_t b = (uint32_t)(q < 0 ? -q : q), mask = q < 0 ? 0u : 0xffffffffu;
    if (k == 0) {  // R 4, R 2^32 after it
#pragma unroll
      for (int i = W - 1; i > 0; --i) R[i] = funnel_l(R[i - 1], R[i], 2);
      R[0] <<= 2;
    } else {
#pragma unroll
      for (int i = W - 1; i > 0; --i) R[i] = R[i - 1];
      R[0] = 0u;
    }
    uint32_t P[W + 1], O[W + 1];  // b M: even and odd words' products apart
#pragma unroll
    for (int i = 0; i < 2 * N; i += 2) {
      const uint64_t e = (uint64_t)M[i] * b, o = (uint64_t)M[i + 1] * b;
      P[i] = (uint32_t)e;
      P[i + 1] = (uint32_t)(e >> 32);
      O[i + 1] = (uint32_t)o;
      O[i + 2] = (uint32_t)(o >> 32);
    }
    P[W - 1] = O[0] = 0u;
    add_words<W>(P, O, 0u);
#pragma unroll
    for (int i = 0; i < W; ++i) P[i] ^= mask;  // R - q M
    add_words<W>(R, P, mask & 1u);
    if (k > 0) {  // Q = Q 2^32 + q
#pragma unroll
      for (int i = W - 1; i > 0; --i) Q[i] = Q[i - 1];
      Q[0] = 0u;
    }
    const uint32_t up = q < 0 ? 0xffffffffu : 0u;
#pragma unroll
    for (int i = 1; i < W; ++i) O[i] = up;
    O[0] = (uint32_t)q;
    add_words<W>(Q, O, 0u);
  }
  if (R[W - 1] >> 31) {
    uint32_t D[W];
#pragma unroll
    for (int i = 0; i < W; ++i) D[i] = i < 2 * N ? M[i < 2 * N ? i : 0] : 0u;
    add_words<W>(R, D, 0u);
    uint32_t one[W] = {1u};
    sub_words<W>(Q, one);
  }
  return !is_zero<W>(R);
}
// (Q + sticky) 2^scale rounded, sticky below Q's last bit.
template <int N>
MPD_FN Val<N> round_quotient(const uint32_t* Q, bool sticky, bool neg, long long scale) {
  constexpr int K = 2 * N + 2;
  uint32_t S[K];
  S[0] = sticky ? 1u : 0u;
#pragma unroll
  for (int i = 0; i < 2 * N + 1; ++i) S[i + 1] = Q[i];
  const int sh = normalize<K>(S);
  return round_top<N, K>(S, neg, scale - 32 - sh);
}

// 1 / d: Q = floor(2^K / M_d), K = 128N + 2, remainder sticky.
template <int N>
MPD_CALL Val<N> recip(Val<N> d) {
  uint32_t Q[2 * N + 1], R[2 * N + 1];
#pragma unroll
  for (int i = 0; i < 2 * N; ++i) R[i] = 0u;
  R[2 * N] = 1u;
  const bool sticky = long_division<N>(R, d.m, Q);
  return round_quotient<N>(Q, sticky, d.neg, -(128LL * N + 2) - d.s);
}

// a / b: Q = floor(M_a 2^K / M_b), K = 64N + 2, remainder sticky.  b must be nonzero.
template <int N>
MPD_CALL Val<N> divide(Val<N> a, Val<N> b) {
  if (a.zero) return zero_val<N>();
  uint32_t Q[2 * N + 1], R[2 * N + 1];
#pragma unroll
  for (int i = 0; i < 2 * N; ++i) R[i] = a.m[i];
  R[2 * N] = 0u;
  const bool sticky = long_division<N>(R, b.m, Q);
  return round_quotient<N>(Q, sticky, a.neg != b.neg, a.s - b.s - (64LL * N + 2));
}

// sqrt(a), a >= 0: Y = floor(sqrt(M 2^e)), the radicand 2 (64N + 2) bits wide (e even with s - e),
// remainder sticky.
template <int N>
MPD_CALL Val<N> root(Val<N> a) {
  if (a.zero) return a;
  long long e = 64LL * N + 4;
  if ((a.s - e) & 1) e += 1;
  Val<N> x = a;  // M 2^e
  x.neg = false;
  x.s = e;
  const Val<N> y = mul<N>(x, rsqrt_approx<N>(x));  // ~ sqrt(M 2^e)
  uint32_t Y[2 * N + 1], R[2 * N + 2], D[2 * N + 2];
  to_words<N>(y, 0, Y);
  {  // R = M 2^e - Y^2 modulo 2^(64N + 64)
    const int r = (int)(e - 64LL * N);
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) R[i] = 0u;
    R[2 * N] = a.m[0] << r;
    R[2 * N + 1] = funnel_l(a.m[0], a.m[1], r);
    sub_product<N>(R, Y, Y);  // Y (Y mod 2^64N), the rest of Y^2 follows
    const uint64_t t0 = (uint64_t)Y[2 * N] * Y[0];
    const uint32_t up[2] = {(uint32_t)t0, (uint32_t)(t0 >> 32) + Y[2 * N] * Y[1]};
    sub_words<2>(R + 2 * N, up);
  }
  // 0 <= R <= 2Y: while negative Y -= 1, R += 2Y + 1 (new Y); while R > 2Y, R -= 2Y + 1, Y += 1
  auto twice = [&]() {  // D = 2Y + 1
    D[0] = (Y[0] << 1) | 1u;
#pragma unroll
    for (int i = 1; i < 2 * N + 1; ++i) D[i] = funnel_l(Y[i - 1], Y[i], 1);
    D[2 * N + 1] = Y[2 * N] >> 31;
  };
#pragma unroll 1
  for (int it = 0; it < 4096 && (R[2 * N + 1] >> 31); ++it) {
    uint32_t one[2 * N + 1] = {1u};
    sub_words<2 * N + 1>(Y, one);
    twice();
    add_words<2 * N + 2>(R, D, 0u);
  }
#pragma unroll 1
  for (int it = 0; it < 4096; ++it) {
    twice();
    if (cmp_words<2 * N + 2>(R, D) < 0) break;
    sub_words<2 * N + 2>(R, D);
    add_word<2 * N + 1>(Y, 1u);
  }
  return round_quotient<N>(Y, !is_zero<2 * N + 2>(R), false, (a.s - e) / 2);
}

// ---- exact dots ----

// Register accumulator: terms of 128N bits whose scales span at most kSpanBits, 72 bits of room
// for the count and the sign.
template <int N>
struct Acc {
  static constexpr int W = 4 * N + 12;
  uint32_t w[W];
};
constexpr int kSpanBits = 12 * 32 - 72;

template <int N, int Q>
struct PlaceStage {  // T <<= q words, q's bits from Q up
  static MPD_FN void run(uint32_t* T, int q) {
    if (q & Q) {
#pragma unroll
      for (int i = Acc<N>::W - 1; i >= 0; --i) T[i] = i >= Q ? T[i >= Q ? i - Q : 0] : 0u;
    }
    PlaceStage<N, (Q < 8 ? 2 * Q : 0)>::run(T, q);
  }
};
template <int N>
struct PlaceStage<N, 0> {
  static MPD_FN void run(uint32_t*, int) {}
};

// acc += (-1)^neg P 2^sh, P 4N words, 0 <= sh < 512, the shifted P within the accumulator.
template <int N>
MPD_FN void acc_add(Acc<N>& acc, const uint32_t* P, int sh, bool neg) {
  constexpr int W = Acc<N>::W;
  uint32_t T[W];
  const int r = sh & 31;
  T[0] = P[0] << r;
#pragma unroll
  for (int i = 1; i < 4 * N; ++i) T[i] = funnel_l(P[i - 1], P[i], r);
  T[4 * N] = funnel_l(P[4 * N - 1], 0u, r);
#pragma unroll
  for (int i = 4 * N + 1; i < W; ++i) T[i] = 0u;
  PlaceStage<N, 1>::run(T, sh >> 5);
  const uint32_t mask = neg ? 0xffffffffu : 0u;
#pragma unroll
  for (int i = 0; i < W; ++i) T[i] ^= mask;
  add_words<W>(acc.w, T, mask & 1u);
}

// acc += v's mantissa 2^sh with v's sign, 0 <= sh <= kSpanBits + 64N: placed like a product's upper
// half when it sits that high.
template <int N>
MPD_FN void acc_add_value(Acc<N>& acc, const Val<N>& v, long long sh) {
  const bool high = sh >= 64LL * N;
  uint32_t P[4 * N];
#pragma unroll
  for (int i = 0; i < 2 * N; ++i) {
    P[i] = high ? 0u : v.m[i];
    P[2 * N + i] = high ? v.m[i] : 0u;
  }
  acc_add<N>(acc, P, (int)(high ? sh - 64LL * N : sh), v.neg);
}

// acc 2^lo rounded once (acc two's complement, destroyed).
template <int N>
MPD_FN Val<N> acc_round(Acc<N>& acc, long long lo) {
  constexpr int W = Acc<N>::W;
  const bool neg = acc.w[W - 1] >> 31;
  if (neg) neg_words<W>(acc.w);
  if (is_zero<W>(acc.w)) return zero_val<N>();
  const int sh = normalize<W>(acc.w);
  return round_top<N, W>(acc.w, neg, lo - sh);
}

#if defined(__CUDACC__)

// The terms of dot() that span more than kSpanBits: the accumulator in local memory.
template <int N, int G>
__device__ __noinline__ Val<N> dot_wide(const Val<N>* a, const unsigned char* x, long xs, const unsigned char* y,
                                        long ys, int count, int sub, unsigned mask, long long lo, int W) {
  constexpr long esz = 8L * N + 8;
  uint32_t acc[2 * kAccWords];
  for (int w = 0; w < 2 * W; ++w) acc[w] = 0u;
  auto add = [&](const uint32_t* P, int words, long long sh, bool neg) {  // acc += (-1)^neg P 2^sh
    const int q = (int)(sh >> 5), r = (int)(sh & 31);
    const uint32_t m = neg ? 0xffffffffu : 0u;
    uint32_t c = neg ? 1u : 0u, prev = 0u;
    for (int i = 0; q + i < 2 * W; ++i) {
      const uint32_t cur = i < words ? P[i] : 0u;
      const uint64_t t = (uint64_t)acc[q + i] + (funnel_l(prev, cur, r) ^ m) + c;
      acc[q + i] = (uint32_t)t;
      c = (uint32_t)(t >> 32);
      prev = cur;
    }
  };
  if (sub == 0 && a && !a->zero) add(a->m, 2 * N, a->s - lo, a->neg);
#pragma unroll 1
  for (int c = sub; c < count; c += G) {
    const Val<N> xv = load<N>(x + c * xs * esz), yv = load<N>(y + c * ys * esz);
    if (xv.zero || yv.zero) continue;
    uint32_t P[4 * N];
    mul_words<N>(P, xv.m, yv.m);
    add(P, 4 * N, xv.s + yv.s - lo, (xv.neg != yv.neg) != (a != nullptr));
  }
  for (int o = G / 2; o > 0; o >>= 1) {
    uint32_t c = 0;
    for (int w = 0; w < 2 * W; ++w) {
      const uint64_t t = (uint64_t)acc[w] + __shfl_xor_sync(mask, acc[w], o) + c;
      acc[w] = (uint32_t)t;
      c = (uint32_t)(t >> 32);
    }
  }
  const bool neg = acc[2 * W - 1] >> 31;
  if (neg) {
    uint32_t c = 1;
    for (int w = 0; w < 2 * W; ++w) {
      acc[w] = ~acc[w] + c;
      c = (c && acc[w] == 0) ? 1u : 0u;
    }
  }
  int top = 2 * W - 1;
  while (top >= 0 && acc[top] == 0) --top;
  if (top < 0) return zero_val<N>();
  uint32_t S[2 * N + 2];  // the leading 2N + 1 words and a sticky word
  uint32_t low = 0;
#pragma unroll
  for (int i = 0; i < 2 * N + 1; ++i) {
    const int w = top - (2 * N) + i;
    S[i + 1] = w >= 0 ? acc[w] : 0u;
  }
  for (int w = top - 2 * N - 1; w >= 0; --w) low |= acc[w];
  S[0] = low ? 1u : 0u;
  const int sh = normalize<2 * N + 2>(S);
  return round_top<N, 2 * N + 2>(S, neg, lo + 32LL * (top - 2 * N - 1) - sh);
}

// a - sum_c x[c] y[c] (a given) or sum_c x[c] y[c] (a null), the exact value rounded once, by the
// aligned group of G lanes (a power of two; every lane of the group calls with the same
// arguments and gets the result): each lane accumulates the terms c = lane, lane + G, ... exactly in one frame
// (the group's lowest scale), and the partial accumulators are summed exactly by a butterfly.
// x_c at x + c * xs, y_c at y + c * ys (element strides).  *ok = false when the terms do not fit
// kAccWords words.
template <int N, int G>
__device__ __noinline__ Val<N> dot(const Val<N>* a, const unsigned char* x, long xs, const unsigned char* y, long ys,
                                   int count, bool* ok) {
  constexpr long esz = 8L * N + 8;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1);
  const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (lane & ~(G - 1));
  long long lo = LLONG_MAX, hi = LLONG_MIN;
#pragma unroll 1
  for (int c = sub; c < count; c += G) {
    long long sx, sy;
    const bool lx = load_scale<N>(x + c * xs * esz, &sx), ly = load_scale<N>(y + c * ys * esz, &sy);
    if (!lx || !ly) continue;
    const long long s = sx + sy;
    lo = s < lo ? s : lo;
    hi = s > hi ? s : hi;
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const long long l2 = __shfl_xor_sync(mask, lo, o), h2 = __shfl_xor_sync(mask, hi, o);
    lo = l2 < lo ? l2 : lo;
    hi = h2 > hi ? h2 : hi;
  }
  if (a && !a->zero) {  // the addend's top bit sits where a product term's would at scale s - 64N
    lo = a->s < lo ? a->s : lo;
    hi = (a->s - 64LL * N) > hi ? (a->s - 64LL * N) : hi;
  }
  if (lo == LLONG_MAX) return zero_val<N>();
  if (hi - lo > kSpanBits) {
    const long long span = hi - lo + 128LL * N + 72;  // largest term's width + log2(count) + sign
    const long long W = (span + 63) / 64 + 1;
    if (W > kAccWords) {
      *ok = false;
      return zero_val<N>();
    }
    return dot_wide<N, G>(a, x, xs, y, ys, count, sub, mask, lo, (int)W);
  }
  Acc<N> acc;
#pragma unroll
  for (int w = 0; w < Acc<N>::W; ++w) acc.w[w] = 0u;
  uint32_t P[4 * N];
  if (sub == 0 && a && !a->zero) acc_add_value<N>(acc, *a, a->s - lo);
#pragma unroll 1
  for (int c = sub; c < count; c += G) {
    const Val<N> xv = load<N>(x + c * xs * esz), yv = load<N>(y + c * ys * esz);
    if (xv.zero || yv.zero) continue;
    mul_words<N>(P, xv.m, yv.m);
    acc_add<N>(acc, P, (int)(xv.s + yv.s - lo), (xv.neg != yv.neg) != (a != nullptr));
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    uint32_t t[Acc<N>::W];
#pragma unroll
    for (int w = 0; w < Acc<N>::W; ++w) t[w] = __shfl_xor_sync(mask, acc.w[w], o);
    add_words<Acc<N>::W>(acc.w, t, 0u);
  }
  return acc_round<N>(acc, lo);
}

// f(std::integral_constant<int, N>) for a run-time limb count 1..kMaxN (a kernel per limb count).
template <class F>
inline void by_limbs(int N, F&& f) {
  switch (N) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    default: break;
  }
}

#endif  // __CUDACC__

}  // namespace mpd
