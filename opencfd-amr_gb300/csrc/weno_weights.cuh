// The nonlinear weights of the FP64 WENO-Z on the integer pipes.
//
// GB300 executes two FP64 instructions per cycle per SM and 64 to 128 integer
// instructions, so a product of positive numbers as 64-bit integers with separate
// exponents (three 32 x 32 -> 64 bit multiply-adds, a shift and an add) costs a
// fraction of one FP64 multiplication's issue time.  The smoothness indicators are
// sums of two squares and the weights sums and products of them.  Values are m 2^e
// with m below 2^63 and truncated products, between 54 and 62 significant bits at
// every step against FP64's 53, and the division is one by the sum's integer
// reciprocal: the results are rounded to FP64 once.  Against 128-bit arithmetic the
// coefficients' error is 0.5e-16 rms, where the same formulas in FP64 have 0.8e-16 to
// 6e-16; where tau cancels both lose digits, this form six bits fewer.  Exponents are
// integers, so no intermediate overflows or underflows.
// They replace 27 of 37 FP64 operations of a face and side by about 450 integer
// instructions, which run in the FP64 pipe's shadow.  A stage of the 3D blast on
// 128x128x64 cells: 3.32 ms in FP64; 2.38 ms with the weights here; 2.17 ms with
// the division too; 1.91 ms with the indicators too (808 instead of 1630 FP64
// instructions per cell).  With the split's 14 operations less 1.79 ms (750); with the
// correction formed here too, 1.73 ms (649 per cell, the FP64 pipe 65 % busy, 1.49
// instead of 0.37 instructions issued per cycle): the integer chain's latency on 16
// warps per SM now weighs as much as the FP64 pipe.  128-bit arithmetic on faces of
// smooth, random and jumping lines puts the face value's rms error at 0.95 of that of
// FP64 coefficients (smooth, random), 1.0 (jumps).
#pragma once

#include <cstdint>
#include <cstring>

namespace ocfd {
namespace wz {

#if defined(__CUDACC__)
#define OCFD_HD __host__ __device__ __forceinline__
#else
#define OCFD_HD inline
#endif

OCFD_HD uint64_t bits_of(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
OCFD_HD double double_of(uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// x >> s, 0 for s >= 64
OCFD_HD uint64_t shr(uint64_t x, int s) {
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));  // clamps the shift
    return r;
#else
    return s > 63 ? 0 : x >> s;
#endif
}
OCFD_HD int imax(int a, int b) { return a > b ? a : b; }
OCFD_HD int lead_zeros(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}

// floor(a b / 2^64) to within 2 below, a, b < 2^63
OCFD_HD uint64_t mul_hi(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    const uint64_t t = (uint64_t)ah * bl + (uint64_t)al * bh;
    return (uint64_t)ah * bh + (t >> 32);
}
OCFD_HD uint64_t sq_hi(uint64_t a) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    return (uint64_t)ah * ah + (((uint64_t)ah * al) >> 31);
}

struct Num {  // m 2^e
    uint64_t m;
    int e;
};
// m in [2^32, 2^63) shifted up to [2^62, 2^63)
OCFD_HD Num normalise(uint64_t m, int e) {
    const int z = lead_zeros((uint32_t)(m >> 32)) - 1;
    return Num{m << z, e - z};
}
// the double nearest m 2^e (m in [2^62, 2^63)), at least 2^-1022
OCFD_HD double pack(const Num& a) {
    const int x = imax(a.e + 62 + 1022, 0);  // biased exponent - 1: the leading bit adds one
    return double_of(((a.m + 0x200u) >> 10) + ((uint64_t)(uint32_t)x << 52));
}
// about 1/x to FP32 accuracy (the seed below corrects any error up to 2^-20)
OCFD_HD float rcp_seed(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}
// 2^125 / m to within a few units, below 2^63 (m in [2^62, 2^63)): an FP32 seed y of
// relative error e <= 2^-20 and one cubic step y (1 + e + e^2)
OCFD_HD uint64_t recip(uint64_t m) {
    m *= 2;
    const uint32_t mh = (uint32_t)(m >> 32), ml = (uint32_t)m;
    const uint32_t y = (uint32_t)(rcp_seed((float)mh) * 0x1p62f);         // (2^30, 2^31]
    const uint64_t t = (uint64_t)mh * y + (((uint64_t)ml * y) >> 32);     // 2^62 (1 - e)
    const int64_t d = (int64_t)(0x4000000000000000ull - t);              // 2^62 e, 43 bits
    const int32_t dh = (int32_t)(d >> 12);                                // 2^50 e
    const int64_t c = d + (((int64_t)dh * dh) >> 38);                    // 2^62 (e + e^2)
    const int32_t ch = (int32_t)(c >> 22);
    const uint32_t cl = (uint32_t)c & 0x3fffffu;
    return ((uint64_t)y << 32) + (uint64_t)(((int64_t)ch * (int64_t)y) >> 8) + (((uint64_t)cl * y) >> 30) - 8;
}

OCFD_HD bool negative(double x) { return (int64_t)bits_of(x) < 0; }
// |x| as a square's factor: m in [2^62, 2^63), biased exponent
OCFD_HD Num unpack_abs(double x) {
    const uint64_t b = bits_of(x) & 0x7fffffffffffffffull;
    return Num{((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10, (int)(b >> 52)};
}
// Squares stand for m 2^(e - 2106) here.  12 eps + 13 e^2 of a second difference e,
// the part of 12 (eps + beta) that belongs to a triple of cells (eps = 1e-6)
constexpr uint64_t kEps12 = 0x192a737110e45380ull;  // 12 eps = kEps12 2^-77
constexpr int kEps12Exp = 2106 - 77;
OCFD_HD Num curvature(double e) {
    const Num a = unpack_abs(e);
    const int x = 2 * a.e + 5;
    return Num{shr((sq_hi(a.m) >> 5) * 13, imax(kEps12Exp - x, 0)) + shr(kEps12, imax(x - kEps12Exp, 0)),
               imax(x, kEps12Exp)};  // [2^58, 2^62)
}
// D = 12 (eps + beta) = 3 g^2 + (12 eps + 13 e^2), m in [2^62, 2^63)
OCFD_HD Num indicator(double g, const Num& c) {
    const Num a = unpack_abs(g);
    const int x = 2 * a.e + 2;
    return normalise(shr((sq_hi(a.m) >> 2) * 3, imax(c.e - x, 0)) + shr(c.m, imax(x - c.e, 0)), imax(x, c.e));
}
// |a - b|, m in [2^62, 2^63), or 0 with an exponent whose double lies below every
// indicator's, so that the square aligns nothing else away (an exponent next to a's,
// as cancelled digits leave it, shifted the middle indicator out where the outer two
// are equal and 2^62 times larger)
OCFD_HD Num difference(const Num& a, const Num& b) {
    const int x = imax(a.e, b.e);
    const int64_t d = (int64_t)(shr(a.m, x - a.e) - shr(b.m, x - b.e));
    const uint64_t m = (uint64_t)(d < 0 ? -d : d);
    const int z = ((m >> 32) ? lead_zeros((uint32_t)(m >> 32)) : 32 + lead_zeros((uint32_t)m | 1u)) - 1;
    return Num{m << z, m ? x - z : x - 8192};
}

// The weights of the three candidates' second differences: with D_k = 12 (eps +
// beta_k) from the first differences g_k = 2 sqrt(beta_k - 13/12 e_k^2) and the
// curvature terms of the three sub-stencils, tau = |D_1 - D_3|, q_k = D_k^2 and
// A_k = q_i q_j (q_k + tau^2) ({i, j} the other two), b = (A_1, 6 A_2, 3 A_3) and
// 1 / (3 (b1 + b2 + b3)) = z 2^(-125 - e).
struct Weights {
    Num b1, b2, b3;
    uint64_t z;
    int e;
};
OCFD_HD Weights weights(double g1, double g2, double g3, const Num& k1, const Num& k2, const Num& k3) {
    const Num d1 = indicator(g1, k1), d2 = indicator(g2, k2), d3 = indicator(g3, k3), t = difference(d1, d3);
    const uint64_t q1 = sq_hi(d1.m), q2 = sq_hi(d2.m), q3 = sq_hi(d3.m), tt = sq_hi(t.m);  // [2^60, 2^62)
    const int e1 = 2 * d1.e, e2 = 2 * d2.e, e3 = 2 * d3.e, et = 2 * t.e;
    // q_k + tau^2 at the larger exponent
    const uint64_t s1 = shr(q1, imax(et - e1, 0)) + shr(tt, imax(e1 - et, 0));
    const uint64_t s2 = shr(q2, imax(et - e2, 0)) + shr(tt, imax(e2 - et, 0));
    const uint64_t s3 = shr(q3, imax(et - e3, 0)) + shr(tt, imax(e3 - et, 0));  // [2^60, 2^63)
    const uint64_t r23 = mul_hi(2 * q2, 2 * q3) * 2, r13 = mul_hi(2 * q1, 2 * q3) * 2, r12 = mul_hi(2 * q1, 2 * q2) * 2;
    // A_k in [2^55, 2^62); the constant exponent offsets are common to all three
    Weights w;
    w.b1 = normalise(mul_hi(r23, s1), e2 + e3 + imax(e1, et));
    w.b2 = normalise(3 * (mul_hi(r13, s2) >> 1), e1 + e3 + imax(e2, et) + 2);  // 6 A_2
    w.b3 = normalise(3 * (mul_hi(r12, s3) >> 1), e1 + e2 + imax(e3, et) + 1);  // 3 A_3
    const int top = imax(w.b1.e, imax(w.b2.e, w.b3.e)) + 4;
    const Num s =
        normalise(3 * (shr(w.b1.m, top - w.b1.e) + shr(w.b2.m, top - w.b2.e) + shr(w.b3.m, top - w.b3.e)), top);  // 3 s
    w.z = recip(s.m);
    w.e = s.e;
    return w;
}

// The correction (b1 e1 + b2 e2 + b3 h / 2) / (3 s), h = 3 e2 - e3, to the face value
// V3 + d2 / 2, rounded once.  The products are aligned to the largest of them, so
// what is cut off stays below 2^-57 of it; factors below 2^-1022 count as zero, and
// the result is not a number if one of them is not finite.
OCFD_HD double correction(const Weights& w, double e1, double e2, double h) {
    const Num a1 = unpack_abs(e1), a2 = unpack_abs(e2), a3 = unpack_abs(h);
    const int big = imax(a1.e, imax(a2.e, a3.e));
    if (big == 0) return 0.0;
    const int x1 = w.b1.e + a1.e, x2 = w.b2.e + a2.e, x3 = w.b3.e - 1 + a3.e;
    const int top = imax(x1, imax(x2, x3)) + 1;
    const int64_t p1 = (int64_t)shr(mul_hi(w.b1.m, a1.m), top - x1), p2 = (int64_t)shr(mul_hi(w.b2.m, a2.m), top - x2),
                  p3 = (int64_t)shr(mul_hi(w.b3.m, a3.m), top - x3);  // below 2^61 each
    const int64_t sum = (negative(e1) ? -p1 : p1) + (negative(e2) ? -p2 : p2) + (negative(h) ? -p3 : p3);
    const uint64_t m = (uint64_t)(sum < 0 ? -sum : sum);
    const int z = ((m >> 32) ? lead_zeros((uint32_t)(m >> 32)) : 32 + lead_zeros((uint32_t)m | 1u)) - 1;
    // |e_k| = a.m 2^(a.e - 1085), a product's high half 2^64, z 2^-125 and its high half 2^64
    const double c = pack(normalise(mul_hi(m << z, w.z), top - z - w.e - 1085 + 64 - 61));
    if (m == 0 || big == 0x7ff) return big == 0x7ff ? double_of(0x7ff8000000000000ull) : 0.0;
    return double_of(bits_of(c) | ((uint64_t)sum & 0x8000000000000000ull));
}

}  // namespace wz
}  // namespace ocfd
