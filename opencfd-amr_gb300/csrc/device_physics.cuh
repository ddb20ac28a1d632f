// Point-level physics of the ideal-gas path, written for the GPU (and callable
// on the host: include/ocfd/compat.H builds the reference's per-point functions
// from them).  Each function keeps the operation order of the reference
// expression it replaces,
// so the FP64 kernels agree with the reference to rounding (the parity tests
// use 1e-12 norm-wise; differences come only from FMA contraction).
#pragma once

#include "ocfd_internal.h"
#include "weno_weights.cuh"

namespace ocfd {

enum { URHO = 0, UMX = 1, UMY = 2, UMZ = 3, UEDEN = 4, NCONS = 5 };
enum { QRHO = 0, QU = 1, QV = 2, QW = 3, QPRES = 4, QT = 5, QC = 6, QGAMA = 7 };

__host__ __device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }
__host__ __device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }

// c2prim, Source/kernel/Kernels.H:13-40.  q = rho, u, v, w, p, T, c.
__host__ __device__ __forceinline__ void c2prim_ideal(const DevParm& P, double u0, double u1, double u2,
                                             double u3, double u4, double* q) {
    double rho = dmax(u0, P.smallr);
    double rhoinv = 1.0 / rho;
    double ux = u1 * rhoinv, uy = u2 * rhoinv, uz = u3 * rhoinv;
    double kineng = 0.5 * (ux * ux + uy * uy + uz * uz);
    double ei = u4 - rho * kineng;
    double p = dmax((P.gamma - 1.0) * ei, P.smallp);
    double T = p / (rho * P.Rg);
    q[QRHO] = rho;
    q[QU] = ux;
    q[QV] = uy;
    q[QW] = uz;
    q[QPRES] = p;
    q[QT] = T;
    q[QC] = sqrt(P.gamma * P.Rg * T);
}

// Steger-Warming split along D (Source/kernel/FluxSplit.H:11-193), given the
// split constants t1 = 1/(2g), t2 = 2(g-1), t3 = (3-g)/(2(g-1)), gm1 = g-1.
// T = double keeps the reference's expressions; T = float serves the
// mixed-precision form.
template <int D, class T = double>
__host__ __device__ __forceinline__ void sw_split(T d, T u, T v, T w, T c, T t1, T t2, T t3, T gm1, T* fp,
                                         T* fm) {
    const T vel[3] = {u, v, w};
    const T un = vel[D];
    const T uc1 = un - c, uc2 = un + c;
    T a0 = u, a1 = v, a2 = w, b0 = u, b1 = v, b2 = w;
    if (D == 0) { a0 = uc1; b0 = uc2; }
    if (D == 1) { a1 = uc1; b1 = uc2; }
    if (D == 2) { a2 = uc1; b2 = uc2; }
    const T half = T(0.5);
    const T vvc1 = half * (a0 * a0 + a1 * a1 + a2 * a2);
    const T vvc2 = half * (b0 * b0 + b1 * b1 + b2 * b2);
    const T v2 = gm1 * (u * u + v * v + w * w);
    const T w2 = t3 * c * c;
    const T E1 = un, E2 = un - c, E3 = un + c;
    const T E1P = (E1 + fabs(E1)) * half, E2P = (E2 + fabs(E2)) * half, E3P = (E3 + fabs(E3)) * half;
    const T E1M = E1 - E1P, E2M = E2 - E2P, E3M = E3 - E3P;
    const T t0 = d * t1;
    const T sp = t2 * E1P + E2P + E3P, sm = t2 * E1M + E2M + E3M;
    fp[URHO] = t0 * sp;
    fm[URHO] = t0 * sm;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (m == D) {
            fp[UMX + m] = t0 * (t2 * E1P * un + E2P * uc1 + E3P * uc2);
            fm[UMX + m] = t0 * (t2 * E1M * un + E2M * uc1 + E3M * uc2);
        } else {
            fp[UMX + m] = t0 * vel[m] * sp;
            fm[UMX + m] = t0 * vel[m] * sm;
        }
    }
    fp[UEDEN] = t0 * (E1P * v2 + E2P * vvc1 + E3P * vvc2 + w2 * (E2P + E3P));
    fm[UEDEN] = t0 * (E1M * v2 + E2M * vvc1 + E3M * vvc2 + w2 * (E2M + E3M));
}

// WENO-Z, Source/kernel/Reconstruction.H:83-138: f+ stencil at cells i-3..i+1
__host__ __device__ __forceinline__ double wenoz_plus(double V1, double V2, double V3, double V4, double V5) {
    const double eps = 1e-6;
    double s11 = (13.0 / 12.0) * (V1 - 2.0 * V2 + V3) * (V1 - 2.0 * V2 + V3) +
                 0.25 * (V1 - 4.0 * V2 + 3.0 * V3) * (V1 - 4.0 * V2 + 3.0 * V3);
    double s22 = (13.0 / 12.0) * (V2 - 2.0 * V3 + V4) * (V2 - 2.0 * V3 + V4) + 0.25 * (V2 - V4) * (V2 - V4);
    double s33 = (13.0 / 12.0) * (V3 - 2.0 * V4 + V5) * (V3 - 2.0 * V4 + V5) +
                 0.25 * (3.0 * V3 - 4.0 * V4 + V5) * (3.0 * V3 - 4.0 * V4 + V5);
    double s55 = fabs(s11 - s33);
    s11 = 1.0 + (s55 / (eps + s11)) * (s55 / (eps + s11));
    s22 = 1.0 + (s55 / (eps + s22)) * (s55 / (eps + s22));
    s33 = 1.0 + (s55 / (eps + s33)) * (s55 / (eps + s33));
    double a1 = s11, a2 = 6.0 * s22, a3 = 3.0 * s33;
    double invsum = 1.0 / (a1 + a2 + a3);
    double v1 = 2.0 * V1 - 7.0 * V2 + 11.0 * V3;
    double v2 = -V2 + 5.0 * V3 + 2.0 * V4;
    double v3 = 2.0 * V3 + 5.0 * V4 - V5;
    return (1.0 / 6.0) * invsum * (a1 * v1 + a2 * v2 + a3 * v3);
}

// ... and the mirrored f- stencil at cells i-2..i+2
__host__ __device__ __forceinline__ double wenoz_minus(double V1, double V2, double V3, double V4, double V5) {
    const double eps = 1e-6;
    double s11 = (13.0 / 12.0) * (V5 - 2.0 * V4 + V3) * (V5 - 2.0 * V4 + V3) +
                 0.25 * (V5 - 4.0 * V4 + 3.0 * V3) * (V5 - 4.0 * V4 + 3.0 * V3);
    double s22 = (13.0 / 12.0) * (V2 - 2.0 * V3 + V4) * (V2 - 2.0 * V3 + V4) + 0.25 * (V4 - V2) * (V4 - V2);
    double s33 = (13.0 / 12.0) * (V3 - 2.0 * V2 + V1) * (V3 - 2.0 * V2 + V1) +
                 0.25 * (3.0 * V3 - 4.0 * V2 + V1) * (3.0 * V3 - 4.0 * V2 + V1);
    double s55 = fabs(s11 - s33);
    s11 = 1.0 + (s55 / (eps + s11)) * (s55 / (eps + s11));
    s22 = 1.0 + (s55 / (eps + s22)) * (s55 / (eps + s22));
    s33 = 1.0 + (s55 / (eps + s33)) * (s55 / (eps + s33));
    double a1 = s11, a2 = 6.0 * s22, a3 = 3.0 * s33;
    double invsum = 1.0 / (a1 + a2 + a3);
    double v1 = 11.0 * V3 - 7.0 * V4 + 2.0 * V5;
    double v2 = -V4 + 5.0 * V3 + 2.0 * V2;
    double v3 = 2.0 * V3 + 5.0 * V2 - V1;
    return (1.0 / 6.0) * invsum * (a1 * v1 + a2 * v2 + a3 * v3);
}

#if defined(__CUDACC__)
// 1/x for a normal, finite, non-zero double, to within about one ulp, without an
// IEEE division: the PTX approximate reciprocal (rcp.approx.ftz.f64, a seed
// good to roughly 20 bits) refined by two Newton-Raphson steps
// r <- r + r (1 - x r), each of which squares the relative error (P. Markstein,
// IBM J. Res. Develop. 34 (1990) 111-119).  GB300 issues few FP64 instructions
// per cycle; this takes one MUFU operation and four FMAs where a correctly
// rounded division takes about twice as many FP64 instructions.  The
// arguments it is used on are sums of squares plus a positive epsilon.
__device__ __forceinline__ double rcp_nr(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

// The same by one cubic step r (1 + e + e^2) from the seed (the third-order iteration of
// Householder's family for the reciprocal; relative error e of the seed, so e^3 is below
// the last bit): three FMAs, within 0.51 ulp where x and 1/x are normal; 0 and infinities
// give NaN.  For the chemistry and transport kernels, whose FP64 pipe is busy with
// reciprocals; the flow's primitives keep rcp_nr's last bits.
__device__ __forceinline__ double rcp_cubic(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// WENO-Z of one split flux (Source/kernel/Reconstruction.H:83-138) in the fewest
// FP64 operations (GB300 issues two FP64 instructions per cycle per SM).  The
// stencil V1..V5 is ordered towards the face (f+: cells i-3..i+1; f-: cells
// i+2..i-2, i.e. wenoz_minus(V1..V5) == wenoz_1rcp(V5, V4, V3, V2, V1)).  With
// the first differences d1..d4 of V1..V5 and the second differences e1 = d2 - d1,
// e2 = d3 - d2, e3 = d4 - d3:
//   - The smoothness indicators are (13/12) e_k^2 + (1/4) g_k^2 with g_1 = 2 d2 + e1,
//     g_2 = d2 + d3, g_3 = 2 d3 - e3; the weights alpha_k = c_k (1 + (tau / D_k)^2),
//     D_k = eps + beta_k, c = (1, 6, 3), are multiplied by the common positive factor
//     (D_1 D_2 D_3)^2, which cancels in alpha_k / sum alpha: with q_k = D_k^2, alpha_k
//     becomes c_k A_k, A_k = q_j q_l (q_k + tau^2) ({j, l} the other two).  All of this
//     is done on the integer pipes (weno_weights.cuh).
//   - The candidate polynomials are V3 + (3 d2 + 2 e1) / 6, V3 + (3 d2 + 2 e2) / 6
//     and V3 + (3 d2 + 3 e2 - e3) / 6, so the face value is
//     V3 + d2 / 2 + (2 A_1 e1 + 12 A_2 e2 + 3 A_3 (3 e2 - e3)) / (6 sum c_k A_k):
//     three products, and the rounding of the weights multiplies second
//     differences only.
// The same value up to rounding (parity tests: 1e-12 per right-hand side), finite
// for flux differences below ~1e150.  Differences and curvature terms belong to
// cells of the line and serve neighbouring faces: 10 FP64 operations per face and
// side in runs of three faces (13 for a face alone).  With indicators and candidates
// formed from the values and all of it in FP64 they were 49 (54), and a stage of the
// 3D blast on 128x128x64 cells took 4.00 ms; this way and with the split of split_side
// below, 1.73 ms.
// Every rounding is written out, so the value does not depend on the code around
// the call.
__device__ __forceinline__ double wenoz_face_d(double V3, double d2, double d3, double e1, double e2, double e3,
                                               const wz::Num& k1, const wz::Num& k2, const wz::Num& k3) {
    const double g1 = __fma_rn(2.0, d2, e1), g2 = __dadd_rn(d2, d3), g3 = __fma_rn(2.0, d3, -e3);
    const double corr = wz::correction(wz::weights(g1, g2, g3, k1, k2, k3), e1, e2, __fma_rn(3.0, e2, -e3));
    return __dadd_rn(__fma_rn(0.5, d2, V3), corr);
}
__device__ __forceinline__ double wenoz_1rcp(double V1, double V2, double V3, double V4, double V5) {
    const double d1 = __dsub_rn(V2, V1), d2 = __dsub_rn(V3, V2), d3 = __dsub_rn(V4, V3), d4 = __dsub_rn(V5, V4);
    const double e1 = __dsub_rn(d2, d1), e2 = __dsub_rn(d3, d2), e3 = __dsub_rn(d4, d3);
    return wenoz_face_d(V3, d2, d3, e1, e2, e3, wz::curvature(e1), wz::curvature(e2), wz::curvature(e3));
}
// one side of faces m = 0, 1, 2 whose stencils (ordered towards the face) are
// a[m s] .. a[(m + 4) s], as a window sliding along the line.  The f+ side of a
// run is a = f+ at the first face's stencil start, s = the pencil stride; its f-
// side is a = f- at (start + 7 s), s = -stride, and yields the faces in reverse
// order.
// FLAT: look for a flat line first - the f- of a supersonic stream, an undisturbed
// state - which has its own value at every face, all its differences being exact
// zeros.  For the inviscid kernels, whose shocks run into undisturbed gas: a step of
// the jet on three levels 59.5 -> 56.9 ms, the tube 2.40 -> 2.34 ms, the blast 5.67 ->
// 5.60 ms; states without such lines lose 0.2 % to the test (the viscous box) to 0.5 %
// (the multispecies box), so those kernels go without.
template <bool FLAT>
__device__ __forceinline__ void wenoz_run3(const double* a, int s, double& o0, double& o1, double& o2) {
    double V3 = a[2 * s], V4 = a[3 * s], V5 = a[4 * s];
    const double V1 = a[0], V2 = a[s];
    if constexpr (FLAT) {
        // the high words of two cells send nearly every other line on
        const auto hi = [](double v) { return (unsigned)__double2hiint(v); };
        const auto lo = [](double v) { return (unsigned)__double2loint(v); };
        const unsigned h = hi(V1), l = lo(V1);
        if (hi(V5) == h) {
            const double V6 = a[5 * s], V7 = a[6 * s];
            const unsigned off = (hi(V2) ^ h) | (lo(V2) ^ l) | (hi(V3) ^ h) | (lo(V3) ^ l) | (hi(V4) ^ h) |
                                 (lo(V4) ^ l) | (lo(V5) ^ l) | (hi(V6) ^ h) | (lo(V6) ^ l) | (hi(V7) ^ h) | (lo(V7) ^ l);
            if (off == 0u && (h & 0x7ff00000u) != 0x7ff00000u) {
                o0 = o1 = o2 = V1;
                return;
            }
        }
    }
    const double d1 = __dsub_rn(V2, V1);
    double d2 = __dsub_rn(V3, V2), d3 = __dsub_rn(V4, V3), d4 = __dsub_rn(V5, V4);
    double e1 = __dsub_rn(d2, d1), e2 = __dsub_rn(d3, d2), e3 = __dsub_rn(d4, d3);
    wz::Num k1 = wz::curvature(e1), k2 = wz::curvature(e2), k3 = wz::curvature(e3);
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {
        const double v = wenoz_face_d(V3, d2, d3, e1, e2, e3, k1, k2, k3);
        if (m == 0) o0 = v;
        else if (m == 1) o1 = v;
        else o2 = v;
        if (m < 2) {
            V3 = V4;
            V4 = V5;
            V5 = a[(m + 5) * s];
            d2 = d3;
            d3 = d4;
            d4 = __dsub_rn(V5, V4);
            e1 = e2;
            e2 = e3;
            e3 = __dsub_rn(d4, d3);
            k1 = k2;
            k2 = k3;
            k3 = wz::curvature(e3);
        }
    }
}
#endif

#if defined(__CUDACC__)
// Steger-Warming split along D (Source/kernel/FluxSplit.H:11-193) for the fused
// FP64 kernels, in fewer FP64 operations than sw_split's reference order.  The side
// of un's sign always takes the eigenvalue un and the outer one (un + c there, un - c
// on the other side); the inner one goes to the other side, or to the same one in
// supersonic flow, where the other side is exactly zero.  So each eigenvalue's mass,
// momentum and energy are formed once and placed by selects, instead of once per
// side with zeros.  vvc1 + w2 and vvc2 + w2 are H -+ un c with the total enthalpy
// H = |u|^2 / 2 + c^2 / (gamma - 1) (hc = 1 / (gamma - 1)); the tangential momentum
// fluxes are the mass flux times the velocity.  27 FP64 operations (30 in
// supersonic flow) against 41 with both sides summed: a stage of
// the 3D blast on 128x128x64 cells 1.90 -> 1.79 ms (808 -> 750 FP64 instructions per
// cell), a viscous box of 61x45x37 cells 340 -> 326 us.
// The same values up to rounding (parity tests: 1e-12 per right-hand side);
// every rounding is written out, so the fluxes of a cell do not depend on the
// code around the call.
struct SplitSide {
    bool up, sup;          // un's side is f+; the inner eigenvalue has un's sign
    double outer, inner;   // eigenvalues
};
__device__ __forceinline__ SplitSide split_side(double un, double c) {
    const double uc1 = __dsub_rn(un, c), uc2 = __dadd_rn(un, c);
    SplitSide e;
    e.up = __double_as_longlong(un) >= 0;
    e.outer = e.up ? uc2 : uc1;
    e.inner = e.up ? uc1 : uc2;
    e.sup = (__double2hiint(e.inner) ^ __double2hiint(un)) >= 0;
    return e;
}
// 0, or not a number where x is not finite: the other side of a supersonic cell, whose
// eigenvalues' positive or negative parts are zeros that the reference multiplies
__device__ __forceinline__ double zero_of(double x) {
    return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
}
template <int D>
__device__ __forceinline__ void sw_split_d(double d, double u, double v, double w, double c, double t1, double t2,
                                           double hc, double gm1, double* fp, double* fm) {
    const double vel[3] = {u, v, w};
    const double un = vel[D], ua = vel[(D + 1) % 3], ub = vel[(D + 2) % 3];
    const SplitSide e = split_side(un, c);
    const double q2 = __fma_rn(un, un, __fma_rn(ub, ub, __dmul_rn(ua, ua)));
    const double H = __fma_rn(0.5, q2, __dmul_rn(__dmul_rn(hc, c), c));
    const double ho = __fma_rn(fabs(un), c, H), hi = __fma_rn(-fabs(un), c, H);
    const double t0 = __dmul_rn(d, t1);
    const double T1 = __dmul_rn(t0, un), To = __dmul_rn(t0, e.outer), A1 = __dmul_rn(t2, T1);
    double rB = __dadd_rn(A1, To);
    double mB = __fma_rn(To, e.outer, __dmul_rn(A1, un));
    double eB = __fma_rn(To, ho, __dmul_rn(T1, __dmul_rn(gm1, q2)));
    double rS = __dmul_rn(t0, e.inner), mS = __dmul_rn(rS, e.inner), eS = __dmul_rn(rS, hi);
    if (e.sup) {
        rB = __dadd_rn(rB, rS);
        mB = __dadd_rn(mB, mS);
        eB = __dadd_rn(eB, eS);
        rS = mS = eS = zero_of(eB);  // eB holds every input
    }
    const auto put = [&](int n, double big, double small) {
        fp[n] = e.up ? big : small;
        fm[n] = e.up ? small : big;
    };
    put(URHO, rB, rS);
    put(UMX + D, mB, mS);
    put(UMX + (D + 1) % 3, __dmul_rn(rB, ua), __dmul_rn(rS, ua));
    put(UMX + (D + 2) % 3, __dmul_rn(rB, ub), __dmul_rn(rS, ub));
    put(UEDEN, eB, eS);
}
#endif

#if defined(__CUDACC__)
// max(a, b) for b > 0 (the density and pressure floors) on the integer pipes:
// a double's bits read as a signed integer order as the double does against a
// positive b, a negative a or -0 reading below it (NaN a is the only case that
// differs from a > b ? a : b)
__device__ __forceinline__ double max_floor(double a, double b) {
    return __double_as_longlong(a) > __double_as_longlong(b) ? a : b;
}

// c2prim (Source/kernel/Kernels.H:13-40) for the fused FP64 kernels, in fewer
// FP64 operations: the two divisions become one reciprocal of rho
// (T = p (1/rho) (1/Rg), 1/Rg formed once on the host), the floors are integer
// compares, rho |u|^2 is formed as the momenta times the velocities, and
// c^2 = gamma Rg T as gamma p (1/rho); the same values to within a few ulps.
__device__ __forceinline__ void c2prim_ideal_fast(const DevParm& P, double u0, double u1, double u2, double u3,
                                                  double u4, double* q) {
    const double rho = max_floor(u0, P.smallr);
    const double rhoinv = rcp_nr(rho);
    const double ux = u1 * rhoinv, uy = u2 * rhoinv, uz = u3 * rhoinv;
    const double ei = fma(-0.5, fma(u3, uz, fma(u2, uy, u1 * ux)), u4);
    const double p = max_floor((P.gamma - 1.0) * ei, P.smallp);
    q[QRHO] = rho;
    q[QU] = ux;
    q[QV] = uy;
    q[QW] = uz;
    q[QPRES] = p;
    q[QT] = p * rhoinv * P.invRg;
    q[QC] = sqrt(P.gamma * p * rhoinv);
}
#endif

__host__ __device__ __forceinline__ double sutherland(const DevParm& P, double T) {
    return P.C_s * T * sqrt(T) / (T + P.T_s);
}

}  // namespace ocfd
