// Chinese-remainder reconstruction of the modular Ozaki scheme, shared by the
// CRT kernels of the single call (ozaki2.cu) and the batch (grouped.cu).
#pragma once

#include <cstdint>

namespace phpc {

constexpr int kCrtMaxModuli = 15;  // M < 2^127: weights in four 32-bit limbs, sums in five
constexpr int kCrtMaxLimbs = 10;   // balanced 13-bit digits of M / m_i (15 moduli: 10)
constexpr int kCrtMinModuli = 8;

// Balanced 13-bit digits of the largest M / m_i for the first n moduli
// (residue.cuh's kModuli); make_table computes the same count from the
// moduli and the launchers check that the two agree.
__host__ __device__ constexpr int crt_digits(int n) {
  constexpr int kDigits[kCrtMaxModuli + 1] = {0, 0, 0, 0, 0, 0, 0, 0, 5, 6, 6, 7, 8, 8, 9, 10};
  return kDigits[n];
}

// What the residue GEMMs store per element and modulus: not the residue r_i
// of the product but t_i = r_i ((M / m_i)^-1 mod m_i) mod m_i, symmetric
// (|t_i| <= 182), as a BF16 value (exact). (A's residue planes carry the
// factor (M / m_i)^-1 mod m_i, so the GEMM's sums are t_i mod m_i.) Then
// sum_i t_i (M / m_i) = y (mod M), so the reconstruction needs no
// per-modulus multiplication.

// Constants of the reconstruction on FP32 limbs (crt_limbs), the floats
// in both lanes of a packed f32x2 operation.
struct CrtLimbs {
  int np;                                 // digits of the largest M / m_i (5 .. 10)
  int pow[3];                             // 1, 2^13, 2^26: factors the compiler must not turn into shifts
                                          // (the multiply-adds run beside the shift and logic pipe)
  float2 cw[3];                           // 2^(13 j) / M rounded to float, j = np - 1, np - 2, np - 3
  float2 P[kCrtMaxModuli][kCrtMaxLimbs];  // balanced 13-bit digits of M / m_i, least significant first
  float2 negM[kCrtMaxLimbs + 1];          // balanced 13-bit digits of M, negated
};

struct CrtTable {
  int n;                          // number of moduli
  uint32_t m[kCrtMaxModuli];      // the moduli
  uint32_t W[kCrtMaxModuli][4];   // CRT weights M / m_i (for the stored t_i mod m_i), little-endian 32-bit limbs
  uint32_t M[4];                  // product of the moduli
  uint32_t Mhalf[4];              // floor(M / 2)
  int qlimb;                      // quotient estimate from limbs qlimb, qlimb + 1 (M >> 32 qlimb in [2^20, 2^52))
  float Minv;                     // 1 / (M >> 32 qlimb) rounded to float
  int fast;                       // 1: every result y has |y| / M <= 1/2 - 1/32 (crt_round's one-step path)
                                  //    for this table's K (grouped problems carry their own flag)
  CrtLimbs L;                     // the same reconstruction on FP32 limbs (one-step path)
};

// c + v * 2^x for a double v and an int x, one rounding (the scaling is exact
// unless the result leaves the normal range).
__device__ __forceinline__ double crt_add_scaled(double c, double v, int x) {
  const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(v));
  const int E = static_cast<int>((bits >> 52) & 0x7FF) + x;
  if (E >= 1 && E <= 2046)
    return c + __longlong_as_double(static_cast<long long>((bits & ~(0x7FFull << 52)) | (static_cast<uint64_t>(E) << 52)));
  return c + ldexp(v, x);
}

// A 128-bit magnitude (hi, lo) rounded once to double, sign applied: returns
// v and sets shift so that the value is v * 2^shift (v an integer-valued
// double).
__device__ __forceinline__ double round_magnitude(uint64_t hi, uint64_t lo, bool neg, int& shift) {
  double v;
  if (hi == 0) {
    v = __ull2double_rn(lo);
    shift = 0;
  } else {
    // round the 128-bit magnitude to 53 bits once: its top 64 bits plus a
    // sticky bit for everything below them, converted with round-to-nearest
    const int lz = __clzll(static_cast<long long>(hi));
    const uint64_t topbits = lz ? (hi << lz) | (lo >> (64 - lz)) : hi;
    const uint64_t rest = lz ? (lo << lz) : lo;
    v = __ull2double_rn(topbits | (rest != 0 ? 1ull : 0ull));
    shift = 64 - lz;
  }
  return neg ? -v : v;
}

// The symmetric representative of acc mod M (acc = sum r_i W_i < 2^13 M, as
// five 32-bit limbs) rounded once to double: returns v and sets shift so that
// the result is v * 2^shift (v an integer-valued double, 0 for a zero result).
__device__ __forceinline__ double crt_round(uint32_t (&l)[5], const CrtTable& T, int fast, int& shift) {
  // acc / M estimated in single precision from the 64 bits at limb qlimb
  // (acc >> 32 qlimb < 2^64, M >> 32 qlimb >= 2^20): absolute error below
  // 2^13 (2^-20 + 3 2^-24) < 0.01.
  // (Limbs chosen with constant indices: an array indexed by a runtime value
  // would live in local memory.)
  uint32_t tlo = l[0], thi = l[1];
  if (T.qlimb >= 1) {
    tlo = l[1];
    thi = l[2];
  }
  if (T.qlimb >= 2) {
    tlo = l[2];
    thi = l[3];
  }
  if (T.qlimb >= 3) {
    tlo = l[3];
    thi = l[4];
  }
  const float est = static_cast<float>((static_cast<uint64_t>(thi) << 32) | tlo) * T.Minv;
  uint32_t x[4];  // magnitude of the result
  bool neg;
  if (fast) {
    // The result y satisfies |y| / M < 1/2 - 1/32 (the table checks it), so
    // q = round(acc / M) is exact and y = acc - q M, computed modulo 2^128,
    // is the symmetric representative itself.
    const uint32_t q = __float2uint_rn(est);
    uint64_t carry = 0;
    uint32_t borrow = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint64_t pm = static_cast<uint64_t>(T.M[w]) * q + carry;
      carry = pm >> 32;
      const uint64_t sub = static_cast<uint64_t>(l[w]) - static_cast<uint32_t>(pm) - borrow;
      x[w] = static_cast<uint32_t>(sub);
      borrow = static_cast<uint32_t>(sub >> 63);
    }
    neg = (x[3] >> 31) != 0;
    if (neg) {  // two's complement negation
      uint32_t c = 1;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint64_t t = static_cast<uint64_t>(~x[w]) + c;
        x[w] = static_cast<uint32_t>(t);
        c = static_cast<uint32_t>(t >> 32);
      }
    }
  } else {
    // q = floor(acc / M) from the estimate, corrected by at most one in
    // either direction, then the symmetric representative.
    const uint32_t q = static_cast<uint32_t>(est);
    uint32_t rr[5];
    uint64_t carry = 0;
    uint32_t borrow = 0;
#pragma unroll
    for (int w = 0; w < 5; ++w) {  // r = acc - q M (160-bit two's complement)
      const uint64_t pm = (w < 4 ? static_cast<uint64_t>(T.M[w]) * q : 0) + carry;
      carry = pm >> 32;
      const uint64_t sub = static_cast<uint64_t>(l[w]) - static_cast<uint32_t>(pm) - borrow;
      rr[w] = static_cast<uint32_t>(sub);
      borrow = static_cast<uint32_t>(sub >> 63);
    }
    if (rr[4] & 0x80000000u) {  // negative: q was one too large, add M back
      uint64_t c2 = 0;
#pragma unroll
      for (int w = 0; w < 5; ++w) {
        const uint64_t t = static_cast<uint64_t>(rr[w]) + (w < 4 ? T.M[w] : 0) + c2;
        rr[w] = static_cast<uint32_t>(t);
        c2 = t >> 32;
      }
    } else {  // r >= M: q was one too small, subtract M
      bool ge = rr[4] != 0;
      if (!ge) {
        ge = true;
#pragma unroll
        for (int w = 3; w >= 0; --w)
          if (rr[w] != T.M[w]) {
            ge = rr[w] > T.M[w];
            break;
          }
      }
      if (ge) {
        uint32_t b2 = 0;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint64_t t = static_cast<uint64_t>(rr[w]) - T.M[w] - b2;
          rr[w] = static_cast<uint32_t>(t);
          b2 = static_cast<uint32_t>(t >> 63);
        }
      }
    }
    // symmetric representative: r > M/2 -> r - M, magnitude M - r
    bool gt_half = false;
#pragma unroll
    for (int w = 3; w >= 0; --w)
      if (rr[w] != T.Mhalf[w]) {
        gt_half = rr[w] > T.Mhalf[w];
        break;
      }
#pragma unroll
    for (int w = 0; w < 4; ++w) x[w] = rr[w];
    neg = gt_half;
    if (gt_half) {
      uint32_t b2 = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint64_t t = static_cast<uint64_t>(T.M[w]) - x[w] - b2;
        x[w] = static_cast<uint32_t>(t);
        b2 = static_cast<uint32_t>(t >> 63);
      }
    }
  }
  return round_magnitude((static_cast<uint64_t>(x[3]) << 32) | x[2], (static_cast<uint64_t>(x[1]) << 32) | x[0], neg,
                         shift);
}

// The CRT of one element from its residues r[i] mod m_i: acc = sum r_i W_i,
// rounded as crt_round (fast: the one-step path, allowed when the product's
// grid leaves the margin CrtTable::fast states).
template <int NMOD>
__device__ __forceinline__ double crt_value(const uint32_t (&rr)[kCrtMaxModuli], const CrtTable& T, int fast,
                                            int& shift) {
  // rr[i] is the stored t_i (BF16 bits); acc = sum_i (t_i mod m_i) (M / m_i),
  // 32-bit limbs accumulated in 64 bits (no overflow: 15 x 2^9 x 2^32 < 2^45)
  uint64_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll
  for (int i = 0; i < NMOD; ++i) {
    const int32_t t = __float2int_rn(__uint_as_float(rr[i] << 16));
    const uint32_t r = static_cast<uint32_t>(t < 0 ? t + static_cast<int32_t>(T.m[i]) : t);
    a0 += static_cast<uint64_t>(r) * T.W[i][0];
    a1 += static_cast<uint64_t>(r) * T.W[i][1];
    a2 += static_cast<uint64_t>(r) * T.W[i][2];
    a3 += static_cast<uint64_t>(r) * T.W[i][3];
  }
  uint32_t l[5];
  uint64_t t = a0;
  l[0] = static_cast<uint32_t>(t);
  t = (t >> 32) + a1;
  l[1] = static_cast<uint32_t>(t);
  t = (t >> 32) + a2;
  l[2] = static_cast<uint32_t>(t);
  t = (t >> 32) + a3;
  l[3] = static_cast<uint32_t>(t);
  l[4] = static_cast<uint32_t>(t >> 32);
  return crt_round(l, T, fast, shift);
}

// A reconstructed integer y = w[0] + w[1] 2^52 + w[2] 2^104, the words signed
// and overlapping (|w[0]|, |w[1]| < 2^63).
struct CrtWords {
  int64_t w[3];
};

__device__ __forceinline__ int64_t mad_wide(int a, int b, int64_t c) {
  int64_t d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// The one-step CRT of 2 PAIRS adjacent elements on FP32 limbs, each pair in the
// two lanes of packed f32x2 operations, all pairs computed in one pass over the
// moduli so that each modulus's constants are read once. w[p][i] holds the stored t_i of pair p for modulus i
// (BF16, its first element in the low 16 bits, the second in the high 16
// bits). Valid when every result satisfies |y| / M <= 1/2 - 1/32
// (CrtTable::fast); gives the y of crt_value, element e = 2 p + lane. Every
// step except the quotient estimate is exact in FP32 (all values are integers
// below 2^24):
//  1. t_i from its bits; sum_i t_i (M / m_i) = y (mod M);
//  2. S_j = sum_i t_i P_ij over the balanced 13-bit digits P_ij of M / m_i
//     (|P_ij| <= 2^12, |S_j| <= 15 182 2^12 < 2^23.5);
//  3. q = round(sum_i t_i / m_i) from the top three limb sums,
//     est = sum_j S_j fl(2^(13 j) / M) (|est| <= 7.5, error below 2^-19; the
//     lower limbs weigh below 2^-27); exact under the fast path's margin;
//  4. Y_j = S_j - q M_j (|Y_j| < 2^23.5), the limbs of y = sum_j Y_j 2^(13 j),
//     converted to integers;
//  5. four limbs make a word (|word| < 2^23.5 (2^39 + 2^26 + ..) < 2^63),
//     by 32 x 32 + 64-bit multiply-adds.
// (The limbs were once carried into small digits in FP32 and assembled and
// rounded in 128-bit integers, 213 of the kernel's 349 issue cycles a warp
// element on the integer pipe, its limit; see crt_round_add for the rounding.)
// NMOD = T.n, the number of moduli; NP = T.L.np = crt_digits(NMOD), the
// number of digits of the largest M / m_i.
template <int NMOD, int PAIRS>
__device__ __forceinline__ void crt_limbs(const uint32_t (&w)[PAIRS][kCrtMaxModuli], const CrtTable& T,
                                          CrtWords (&out)[2 * PAIRS]) {
  constexpr int NP = crt_digits(NMOD);
  const float2 kRound = make_float2(12582912.0f, 12582912.0f), kUnround = make_float2(-12582912.0f, -12582912.0f);
  float2 S[PAIRS][NP];
#pragma unroll
  for (int p = 0; p < PAIRS; ++p)
#pragma unroll
    for (int j = 0; j < NP; ++j) S[p][j] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < NMOD; ++i) {
    float2 t[PAIRS];
#pragma unroll
    for (int p = 0; p < PAIRS; ++p)
      t[p] = make_float2(__uint_as_float(w[p][i] << 16), __uint_as_float(w[p][i] & 0xFFFF0000u));
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const float2 pij = T.L.P[i][j];
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) S[p][j] = __ffma2_rn(t[p], pij, S[p][j]);
    }
  }
#pragma unroll
  for (int p = 0; p < PAIRS; ++p) {
    float2 est = __fmul2_rn(S[p][NP - 1], T.L.cw[0]);
    est = __ffma2_rn(S[p][NP - 2], T.L.cw[1], est);
    est = __ffma2_rn(S[p][NP - 3], T.L.cw[2], est);
    const float2 q = __fadd2_rn(__fadd2_rn(est, kRound), kUnround);
    int Y[2][12];  // the limbs; those above NP are zero
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      if (j <= NP) {
        const float2 y = j < NP ? __ffma2_rn(q, T.L.negM[j], S[p][j]) : __fmul2_rn(q, T.L.negM[NP]);
        Y[0][j] = __float2int_rn(y.x);
        Y[1][j] = __float2int_rn(y.y);
      } else {
        Y[0][j] = Y[1][j] = 0;
      }
    }
#pragma unroll
    for (int l = 0; l < 2; ++l)
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        const int(&y)[12] = Y[l];
        int64_t v = 0;
        if (4 * g + 3 <= NP) v = static_cast<int64_t>(static_cast<uint64_t>(static_cast<uint32_t>(y[4 * g + 3]) << 7) << 32);
        if (4 * g + 2 <= NP) v = mad_wide(y[4 * g + 2], T.L.pow[2], v);
        if (4 * g + 1 <= NP) v = mad_wide(y[4 * g + 1], T.L.pow[1], v);
        if (4 * g <= NP) v = mad_wide(y[4 * g], T.L.pow[0], v);
        out[2 * p + l].w[g] = v;
      }
  }
}

// c + y 2^x for a reconstructed y, |y| <= M (1/2 - 1/32): y rounded once to
// double (to nearest even), the sum rounded once.
//
// y is cut in two, floor(y / 2^s) and the s bits below. Each half becomes a
// double through its bits, the upper one by an exact subtraction of a constant,
// and their sum is y's one rounding:
//  - 8 to 12 moduli (|y| < 2^100.4): s = 52, V = floor(y / 2^52), |V| < 2^48.4;
//    (V - 1) 2^52 and 2^52 + the lower half are exact.
//  - 13 to 15 moduli (|y| < 2^108.6, 2^116.9, 2^125.1): s = 52 + SH, B =
//    floor(y / 2^s), |B| < 2^51; (B - 1) 2^s is exact, and 2^s + the lower half
//    has its low SH bits folded into one sticky bit, which lies below half an
//    ulp of y for |y| >= 2^(SH + 54). Values below 2^84 (a zero, a strong
//    cancellation) are rare and take the first form.
// Three FP64 additions a value: 48 cycles of the SM's FP64 pipe a warp, below
// the 58 that a warp's 42 bytes an element take at DRAM speed with 13 moduli.
// Comparing doubles or converting an int64 costs that pipe as much again, so a
// zero is found by its bits (8 moduli: 142 us with r == 0.0).
//
// The kernel at N = 4096, digits assembled and rounded in 128-bit integers /
// so: 8 moduli 114 us, 116; 9 130, 117; 10 136, 119; 11 148, 124; 12 152, 130; 13
// 160, 132; 14 173, 148; 15 178, 166. (13 at N = 16384 2.8 ms, 2.24; 512-problem
// batch 1.81, 1.59.)
template <int NMOD>
__device__ __forceinline__ double crt_round_add(double c, const CrtWords& y, int x) {
  constexpr int SH = NMOD == 15 ? 23 : NMOD == 14 ? 14 : 6;
  constexpr uint64_t kFold = (1ull << SH) - 1;
  constexpr double kUnit = SH == 23 ? 0x1p75 : SH == 14 ? 0x1p66 : 0x1p58;  // 2^s
  const uint64_t low = static_cast<uint64_t>(y.w[0]) & ((1ull << 52) - 1);
  // y = low + 2^52 mid, from 14 moduli (where that mid passes 64 bits) + 2^104 w[2]
  int64_t mid = y.w[1] + (y.w[0] >> 52), B;
  bool small;
  if (NMOD <= 13) {
    mid += static_cast<int64_t>(static_cast<uint64_t>(y.w[2]) << 52);
    B = mid >> SH;
    small = static_cast<uint32_t>(static_cast<int32_t>(mid >> 32) + 1) <= 1u;
  } else {
    B = (mid >> SH) + static_cast<int64_t>(static_cast<uint64_t>(y.w[2]) << (52 - SH));
    small = static_cast<uint64_t>(B + (1ll << (32 - SH))) < (2ull << (32 - SH));
  }
  double r;
  if (NMOD <= 12 || small) {
    const int64_t V =
        NMOD <= 13 ? mid : static_cast<int64_t>(static_cast<uint64_t>(B) << SH | (static_cast<uint64_t>(mid) & kFold));
    const int64_t top = V + static_cast<int64_t>((1023ull + 104) << 52 | 1ull << 51);
    r = (__longlong_as_double(top) - (0x1.8p104 + 0x1p52)) +
        __longlong_as_double(static_cast<long long>(low | (1023ull + 52) << 52));
    if (__double2hiint(r) == 0) return c + 0.0;
  } else {
    const uint64_t bits = (static_cast<uint64_t>(mid) & kFold) << (52 - SH) | low >> SH | ((low & kFold) != 0 ? 1 : 0);
    const int64_t top = B + static_cast<int64_t>((1023ull + 104 + SH) << 52 | 1ull << 51);
    r = (__longlong_as_double(top) - (0x1.8p52 + 1.0) * kUnit) +
        __longlong_as_double(static_cast<long long>(bits | (1023ull + 52 + SH) << 52));
  }
  return crt_add_scaled(c, r, x);
}

// *c += v * 2^(shift + e): the CRT result of one element applied to C
// (c + 0.0 for a zero result, as an exact product would give).
__device__ __forceinline__ void crt_apply(double* c, double v, int shift_plus_e) {
  *c = v == 0.0 ? *c + 0.0 : crt_add_scaled(*c, v, shift_plus_e);
}

// c + v * 2^(shift + e), the value form of crt_apply.
__device__ __forceinline__ double crt_added(double c, double v, int shift_plus_e) {
  return v == 0.0 ? c + 0.0 : crt_add_scaled(c, v, shift_plus_e);
}

}  // namespace phpc
