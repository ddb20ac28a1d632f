// The nonlinear weights of the FP64 WENO-Z on the integer pipes.
//
// GB300 executes two FP64 instructions per cycle per SM and 64 to 128 integer
// instructions, so a product of positive numbers as 64-bit integers with separate
// exponents (three 32 x 32 -> 64 bit multiply-adds, a shift and an add) costs a
// fraction of one FP64 multiplication's issue time.  The weights are sums and
// products of positive numbers only.  Values are m 2^e with m below 2^63 and
// truncated products, between 55 and 62 significant bits at every step against
// FP64's 53, and the division is one by the sum's integer reciprocal: the results
// are rounded to FP64 once.  Largest relative error 1.5e-16 (rms 0.5e-16) against
// 7.5e-16 (1.1e-16) for the same weights in FP64 arithmetic.  Exponents are
// integers, so no intermediate overflows or underflows.
// It replaces 19 of the 37 FP64 operations of a face and side by about 250 integer
// ones, which run in the FP64 pipe's shadow: a stage of the 3D blast on 128x128x64
// cells 3.32 -> 2.17 ms, the FP64 pipe 82 % busy with 1022 instead of 1630
// instructions per cell and the SM issuing 0.88 instead of 0.37 instructions per
// cycle.  (With the sum's reciprocal and the division in FP64: 2.38 ms.)
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
// a positive double: m in [2^62, 2^63), e its biased exponent (a zero or denormal
// becomes about 2^-1023, far below every square it is added to)
OCFD_HD Num unpack(double x) {
    const uint64_t b = bits_of(x);
    return Num{((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10, (int)(b >> 52)};
}
// m >= 2^32 shifted up to [2^63, 2^64)
OCFD_HD Num normalise(uint64_t m, int e) {
    const int z = lead_zeros((uint32_t)(m >> 32));
    return Num{m << z, e - z};
}
// the double nearest m 2^e (m in [2^63, 2^64)), at least 2^-1022
OCFD_HD double pack(const Num& a) {
    const int x = imax(a.e + 63 + 1022, 0);  // biased exponent - 1: the leading bit adds one
    return double_of((a.m >> 11) + ((a.m >> 10) & 1u) + ((uint64_t)(uint32_t)x << 52));
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
// 2^126 / m to within a few units, below 2^63 (m in [2^63, 2^64)): an FP32 seed y of
// relative error e <= 2^-20 and one cubic step y (1 + e + e^2)
OCFD_HD uint64_t recip(uint64_t m) {
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

// The WENO-Z correction's coefficients: from D_k = eps + beta_k > 0 and tau = |D_1 -
// D_3|, with q_k = D_k^2, A_k = q_i q_j (q_k + tau^2) ({i, j} the other two) and s =
// A_1 + 6 A_2 + 3 A_3: c1 = A_1 / (3 s), c2 = 6 A_2 / (3 s), c3 = 3 A_3 / (6 s).
OCFD_HD void weights(double D1, double D2, double D3, double tau, double& c1, double& c2, double& c3) {
    const Num d1 = unpack(D1), d2 = unpack(D2), d3 = unpack(D3), t = unpack(tau);
    const uint64_t q1 = sq_hi(d1.m), q2 = sq_hi(d2.m), q3 = sq_hi(d3.m), tt = sq_hi(t.m);  // [2^60, 2^62)
    const int e1 = 2 * d1.e, e2 = 2 * d2.e, e3 = 2 * d3.e, et = 2 * t.e;
    // q_k + tau^2 at the larger exponent
    const uint64_t s1 = shr(q1, imax(et - e1, 0)) + shr(tt, imax(e1 - et, 0));
    const uint64_t s2 = shr(q2, imax(et - e2, 0)) + shr(tt, imax(e2 - et, 0));
    const uint64_t s3 = shr(q3, imax(et - e3, 0)) + shr(tt, imax(e3 - et, 0));  // [2^60, 2^63)
    const uint64_t r23 = mul_hi(2 * q2, 2 * q3) * 2, r13 = mul_hi(2 * q1, 2 * q3) * 2, r12 = mul_hi(2 * q1, 2 * q2) * 2;
    // A_k in [2^55, 2^62); the constant exponent offsets are common to all three
    const Num b1 = normalise(mul_hi(r23, s1), e2 + e3 + imax(e1, et));
    const Num b2 = normalise(3 * mul_hi(r13, s2), e1 + e3 + imax(e2, et) + 1);  // 6 A_2
    const Num b3 = normalise(3 * mul_hi(r12, s3), e1 + e2 + imax(e3, et));      // 3 A_3
    const int top = imax(b1.e, imax(b2.e, b3.e)) + 4;
    const Num s = normalise(3 * (shr(b1.m, top - b1.e) + shr(b2.m, top - b2.e) + shr(b3.m, top - b3.e)), top);  // 3 s
    const uint64_t z = recip(s.m);
    // b / (3 s) = (b.m / 2) z 2^-61 2^(b.e - s.e)
    c1 = pack(normalise(mul_hi(b1.m >> 1, z), b1.e - s.e - 61));
    c2 = pack(normalise(mul_hi(b2.m >> 1, z), b2.e - s.e - 61));
    c3 = pack(normalise(mul_hi(b3.m >> 1, z), b3.e - s.e - 62));
}

}  // namespace wz
}  // namespace ocfd
