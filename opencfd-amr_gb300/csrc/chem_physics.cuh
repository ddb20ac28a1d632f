// Li-Dryer H2/O2 thermochemistry and transport on the GPU (device functions).
// Included by exactly one translation unit (chem.cu), which owns c_mech.
//
// The thermodynamic functions keep the operation order of the reference routines they
// replace (Source/CHEM/LiDryer.H, Source/CHEM/ChemViscous.H).  The temperature
// inversion, the reaction rates with their solution, and the transport coefficients are
// regrouped, for the FP64 pipe, as said at each.  log and sqrt are CUDA's, exp in the
// rates is exp_tab; results agree with the CPU build to a few ulps, not bit for bit.
#pragma once

#include "device_physics.cuh"
#include "mechanism.h"

namespace ocfd {

__constant__ MechTables c_mech;

// Quantities derived from the tables once on the host, so that the per-cell
// routines divide less (GB300's FP64 pipe runs a division as ~10 instructions):
//   q3, q5   a2 / 3, a4 / 5 of the internal energy and enthalpy polynomials - the
//            same quotients the expressions form first, so these are bit-identical;
//   inv_mw   1 / W_n, which replaces divisions by W (a rounding of the last bit
//            differs from dividing);
//   uw       per range, coefficient and species: the energy polynomial over W,
//            (a0 - 1, a1 / 2, a2 / 3, a3 / 4, a4 / 5, a5 - a5_low) / W;
//   gp       per range, for H2O, H, O, OH, HO2, H2O2: g/(RT) relative to the
//            elements as H2 and O2, constant, T .. T^4, 1/T and ln T terms;
//   nw       nu W_n for nu = 0 .. 4;
//   a0w      A0_n / W_n.
// What depends on Ru and Patm is a context's own (DevParm): these tables are shared.
struct MechDerived {
    double q3[2][NSP], q5[2][NSP];
    double inv_mw[NSP];
    // e_n(T)/(R T W_n) at the bounds 250 K and 3500 K of the temperature
    // inversion (the mixture energies there are then 9 products)
    double umin_w[NSP], umax_w[NSP];
    double uw[2][6][NSP];
    double gp[2][NSP - 3][7];
    double nw[5][NSP];
    double a0w[NSP];
    // enthalpy polynomials h/R = T (c0 + T (c1 + ...)) + c5 per range, and the
    // species-pair constants of the Wilke rule (j < k): (W_j / W_k)^(1/4),
    // 1 / sqrt(8 + 8 W_k / W_j), W_k / W_j
    double hc[2][6][NSP];
    double wr14[NSP][NSP], wden[NSP][NSP], wkj[NSP][NSP];
};
__constant__ MechDerived c_mder;

// NASA-7 coefficient row of species n for temperature T
__device__ __forceinline__ const double* nasa(double T, int n) {
    return T < 1000 ? c_mech.lo[n] : c_mech.hi[n];
}

// speciesInternalEnergy, LiDryer.H:531-614: e/(RT), tc = {., T, T^2, T^3, T^4}
__device__ __forceinline__ void species_internal_energy(double* e, const double* tc) {
    const double T = tc[1];
    const double invT = 1.0 / T;
#pragma unroll
    for (int n = 0; n < NSP; ++n) {
        if (T < 1000) {
            const double* a = c_mech.lo[n];
            e[n] = a[0] - 1.0 + a[1] / 2.0 * tc[1] + c_mder.q3[0][n] * tc[2] + a[3] / 4.0 * tc[3] +
                   c_mder.q5[0][n] * tc[4];
        } else {
            const double* a = c_mech.hi[n];
            e[n] = a[0] - 1.0 + a[1] / 2.0 * tc[1] + c_mder.q3[1][n] * tc[2] + a[3] / 4.0 * tc[3] +
                   c_mder.q5[1][n] * tc[4] + (a[5] - c_mech.lo[n][5]) * invT;
        }
    }
}

// speciesEnthalpy, LiDryer.H:616-695: h/R [K]
__device__ __forceinline__ void species_enthalpy(double T, double* h) {
    const double tc[5] = {T, T * T, T * T * T, T * T * T * T, T * T * T * T * T};
#pragma unroll
    for (int n = 0; n < NSP; ++n) {
        if (T < 1000) {
            const double* a = c_mech.lo[n];
            h[n] = a[0] * tc[0] + a[1] / 2.0 * tc[1] + c_mder.q3[0][n] * tc[2] + a[3] / 4.0 * tc[3] +
                   c_mder.q5[0][n] * tc[4];
        } else {
            const double* a = c_mech.hi[n];
            h[n] = a[0] * tc[0] + a[1] / 2.0 * tc[1] + c_mder.q3[1][n] * tc[2] + a[3] / 4.0 * tc[3] +
                   c_mder.q5[1][n] * tc[4] + (a[5] - c_mech.lo[n][5]);
        }
    }
}

// CKUBMS, LiDryer.H:697-714: mixture internal energy per volume [J/m^3]
__device__ __forceinline__ double ckubms(double T, const double* rhoi, double Ru) {
    double result = 0;
    const double tc[5] = {0, T, T * T, T * T * T, T * T * T * T};
    double ums[NSP];
    const double RT = Ru * T;
    species_internal_energy(ums, tc);
#pragma unroll
    for (int n = 0; n < NSP; ++n) result += rhoi[n] * ums[n] * c_mder.inv_mw[n];
    return result * RT;
}

// CKCVBS, LiDryer.H:801-815
__device__ __forceinline__ double ckcvbs(double T, const double* rhoi, double Ru) {
    double result = 0;
    const double tc[5] = {0, T, T * T, T * T * T, T * T * T * T};
#pragma unroll
    for (int n = 0; n < NSP; ++n) {
        const double* a = nasa(T, n);
        const double cpor = a[0] + a[1] * tc[1] + a[2] * tc[2] + a[3] * tc[3] + a[4] * tc[4];
        result += (cpor - 1.0) * rhoi[n] * c_mder.inv_mw[n];
    }
    return result * Ru;
}

// CKPY, LiDryer.H:10-18
__device__ __forceinline__ double ckpy(const double* rhoi, double T, double Ru) {
    double YOW = 0;
#pragma unroll
    for (int i = 0; i < NSP; ++i) YOW += rhoi[i] * c_mder.inv_mw[i];
    return Ru * T * YOW;
}

// The Newton loop of GET_T_GIVEN_EY (LiDryer.H:833-888) in the reference's
// operation order, from the starting value t1
__device__ __forceinline__ double newton_reference_order(double ein, const double* rhoi, double Ru, double t1) {
    for (int i = 0; i < 200; ++i) {
        const double e1 = ckubms(t1, rhoi, Ru);
        const double cv = ckcvbs(t1, rhoi, Ru);
        double dt = (ein - e1) / cv;
        if (dt > 100.0) dt = 100.0;
        else if (dt < -100.0) dt = -100.0;
        else if (fabs(dt) < 1e-7) break;
        else if (t1 + dt == t1) break;
        t1 += dt;
    }
    return t1;
}

// GET_T_GIVEN_EY, LiDryer.H:833-888: bounded Newton for T from e on NASA-7.
// The mixture energy sum_n rho_n e_n(T) / W_n is one polynomial in T per
// temperature range: its six coefficients are summed once (and again where an
// iterate crosses 1000 K), so an iteration takes one Horner scheme with its
// derivative (10 FMAs) instead of nine species' polynomials (about 190 FP64
// operations of e and cv).  The same iterates up to rounding (some 1e-12 K).  The
// reference drops a last step below 1e-7 K, so where that rounding decides - a step
// within 1e-11 K of the tolerance, one cell in 1e5 or so - the loop is run again in
// the reference's order and both end on the same iterate.  The step's tests are
// integer compares of |dt|'s bits (FP64 compares run on the FP64 pipe); a NaN passes
// them as it passes the reference's.
__device__ __forceinline__ double get_t_given_ey(double e, const double* rhoi, const DevParm& P) {
    const double Ru = P.Ru;
    const int maxiter = 200;
    const double ein = e, tmin = 250, tmax = 3500;
    double smin = 0, smax = 0, As = 0;
#pragma unroll
    for (int n = 0; n < NSP; ++n) {
        smin += rhoi[n] * c_mder.umin_w[n];
        smax += rhoi[n] * c_mder.umax_w[n];
        As += rhoi[n] * c_mder.a0w[n];
    }
    const double emin = smin * (Ru * tmin), emax = smax * (Ru * tmax);
    if (ein < emin) return tmin - (emin - ein) / ckcvbs(tmin, rhoi, Ru);
    if (ein > emax) return tmax - (emax - ein) / ckcvbs(tmax, rhoi, Ru);
    const double es = ein * P.inv_ru;  // e / Ru
    double t1 = es * rcp_cubic(As);
    if (t1 < tmin || t1 > tmax) t1 = tmin + (tmax - tmin) / (emax - emin) * (ein - emin);
    const long long mag = 0x7fffffffffffffffLL;
    const double t0 = t1;
    int h = -1;
    double C[6];
    for (int i = 0; i < maxiter; ++i) {
        const int ht = t1 < 1000 ? 0 : 1;
        if (ht != h) {
            h = ht;
#pragma unroll
            for (int k = 0; k < 6; ++k) C[k] = rhoi[0] * c_mder.uw[h][k][0];
#pragma unroll
            for (int n = 1; n < NSP; ++n)
#pragma unroll
                for (int k = 0; k < 6; ++k) C[k] = fma(rhoi[n], c_mder.uw[h][k][n], C[k]);
        }
        // (e / Ru)(T) = C5 + T (C0 + T (C1 + ...)) and its derivative
        double b = C[4], d = C[4];
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            b = fma(b, t1, C[k]);
            d = fma(d, t1, b);
        }
        b = fma(b, t1, C[5]);
        double dt = (es - b) * rcp_cubic(d);
        const long long m = __double_as_longlong(dt) & mag;
        if (m > 0x4059000000000000LL) {  // |dt| > 100 (or NaN)
            if (dt > 100.0) dt = 100.0;
            else if (dt < -100.0) dt = -100.0;
        } else if (m < 0x3E7AD8A286BBBB13LL) {  // |dt| < 1e-7 + 1e-11
            if (m > 0x3E7AD742AEBDA37DLL) return newton_reference_order(ein, rhoi, Ru, t0);  // > 1e-7 - 1e-11
            break;
        }
        t1 += dt;
    }
    return t1;
}

// exp(x) in 11 FP64 operations (CUDA's takes about 16): P. T. P. Tang's
// table-driven method (ACM Trans. Math. Softw. 15 (1989) 144-157).  x = (k ln 2) /
// 128 + r, |r| <= ln 2 / 256, exp(x) = 2^(k div 128) T_j (1 + p(r)) with j = k mod
// 128, T_j = 2^(j/128) as a sum of two doubles and p the Taylor polynomial of
// degree 5 (its remainder is below 6e-19).  The error is below 0.52 ulp.  Outside
// |x| <= 708 (overflow, denormal results, NaN) CUDA's exp answers.
__device__ const double2 kExp2Tab[128] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54},
    {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56}, {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57}, {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54},
    {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59}, {0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58},
    {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54}, {0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54},
    {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55}, {0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54},
    {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55}, {0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55},
    {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55}, {0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59},
    {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54}, {0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55},
    {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54}, {0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54},
    {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56}, {0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54},
    {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58}, {0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54},
    {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56}, {0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54}, {0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55},
    {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54}, {0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60},
    {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54}, {0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55},
    {0x1.6623882552225p+0, -0x1.bb60987591c34p-54}, {0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56},
    {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57}, {0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54},
    {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54}, {0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54},
    {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56}, {0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55},
    {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54}, {0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56},
    {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55}, {0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56},
    {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54}, {0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56},
    {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54}, {0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54},
    {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54}, {0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54},
    {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57}, {0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54},
    {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55}, {0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54},
    {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54}, {0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55},
    {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54}, {0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54},
    {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54}, {0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54},
    {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55}, {0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54},
    {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54}, {0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54},
    {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}, {0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57}};
__device__ __forceinline__ double exp_tab(double x) {
    if ((__double2hiint(x) & 0x7fffffff) > 0x40862000) return exp(x);
    const double magic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the rounded integer
    const double t = __fma_rn(x, 0x1.71547652b82fep+7, magic);
    const int k = __double2loint(t);
    const double kd = __dsub_rn(t, magic);
    const double2 T = __ldg(&kExp2Tab[k & 127]);
    const double r = __fma_rn(-kd, 0x1.abc9e3b39803fp-63, __fma_rn(-kd, 0x1.62e42fefa39efp-8, x));
    const double q = __fma_rn(__fma_rn(__fma_rn(r, 1.0 / 120.0, 1.0 / 24.0), r, 1.0 / 6.0), r, 0.5);
    const double p = __fma_rn(__dmul_rn(r, r), q, r);
    const double v = __dadd_rn(T.x, __fma_rn(T.x, p, T.y));
    return __hiloint2double(__double2hiint(v) + ((k >> 7) << 20), __double2loint(v));
}

// ------------------------------------------------------------ production rates
// vproductionRate and gauss (LiDryer.H:156-529, 890-942) of one cell, fused: the
// augmented system (I - dt W J W^-1 | dt W wdot) of the substep is accumulated
// reaction by reaction in registers and solved there.  What bounds it is the
// FP64 pipe (two instructions per cycle per SM), so it is written for the fewest
// FP64 operations; integer and select instructions are an order of magnitude
// cheaper.  Against the reference's expressions:
//   - Equilibrium constants.  Every reaction conserves H and O, so Gibbs energies
//     relative to H2 and O2, g'_n = g_n - (H_n / 2) g_H2 - (O_n / 2) g_O2, give
//     the same reaction differences.  With E_n = exp(g'_n) and z_n = c_n E_n, a
//     reaction's rates are k' prod z (reactants) and (Ru T / Patm)^dn k' prod z
//     (products), k' = k / prod E (reactants): six exponentials and reciprocals
//     (g'_H2 = g'_O2 = 0) for the nineteen reactions.
//   - d(rate)/dc_n = nu rate / (c_n + 1e-20): one reciprocal per species.
//   - N2 takes part in no reaction: its row and column are the identity's, its
//     increment is zero, and the system solved has the other eight species.
//   - dt / W_n multiplies the reciprocals and nu W_l is a constant, so each
//     Jacobian term is one FMA into the system's matrix.
//   - Pivot search on the bits of |U| (integer), rows exchanged by selects,
//     the pivot's reciprocal kept for the back substitution.
// 6073 -> 1678 FP64 instructions per cell-substep, the FP64 pipe 88 % busy either
// way: one substep of a 64^3 box 3025 -> 840 us, one step of a reacting 64^3 cube
// (mixed form, 8 substeps; with the faces and transport below) 30.6 -> 9.6 ms.  238-250 registers and no shared
// memory (the 90-double matrix per thread was in shared memory): two CTAs of 128
// threads per SM either way.
constexpr int NRE = NSP - 1;  // reacting species (all but N2)

struct Stoich {
    int s[4];   // distinct species of the reaction (-1 = unused)
    int vf[4];  // forward stoichiometric coefficients of s[]
    int vr[4];  // reverse
};

// reaction with rates wf, wr: right-hand side (column NRE) and matrix; inv[n] =
// dt / ((c_n + eps) W_n)
__device__ __forceinline__ void rxn_accum(const Stoich& X, double wf, double wr, const double* inv,
                                          double (&U)[NRE][NRE + 1]) {
    const double net = wf - wr;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (X.s[a] < 0) continue;
        const int nu = X.vr[a] - X.vf[a];
        const double w = c_mder.nw[nu < 0 ? -nu : nu][X.s[a]];
        U[X.s[a]][NRE] = fma(nu < 0 ? -net : net, w, U[X.s[a]][NRE]);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        if (X.s[b] < 0) continue;
        const int n = X.s[b];
        // a species stands on one side of each reaction
        const int v = X.vf[b] - X.vr[b];
        const double d = (v > 0 ? wf : wr) * inv[n];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (X.s[a] < 0) continue;
            const int c = v * (X.vr[a] - X.vf[a]);  // d(net nu_a)/dc_n = c d; the matrix is I - ...
            const double w = c_mder.nw[c < 0 ? -c : c][X.s[a]];
            U[X.s[a]][n] = fma(c < 0 ? d : -d, w, U[X.s[a]][n]);
        }
    }
}

// columns C.. of the partial-pivot elimination (a template per column: the
// matrix stays in registers)
template <int C>
__device__ __forceinline__ void eliminate(double (&U)[NRE][NRE + 1], double (&ip)[NRE]) {
    const long long mag = 0x7fffffffffffffffLL;
    int pv = C;
    long long best = __double_as_longlong(U[C][C]) & mag;
#pragma unroll
    for (int i = C + 1; i < NRE; ++i) {
        const long long a = __double_as_longlong(U[i][C]) & mag;
        if (a > best) {
            best = a;
            pv = i;
        }
    }
#pragma unroll
    for (int i = C + 1; i < NRE; ++i) {
        const bool sw = pv == i;
#pragma unroll
        for (int j = C; j <= NRE; ++j) {
            const double t = U[C][j];
            U[C][j] = sw ? U[i][j] : t;
            U[i][j] = sw ? t : U[i][j];
        }
    }
    ip[C] = rcp_cubic(U[C][C]);
#pragma unroll
    for (int i = C + 1; i < NRE; ++i) {
        const double m = U[i][C] * ip[C];
#pragma unroll
        for (int j = C + 1; j <= NRE; ++j) U[i][j] = fma(-m, U[C][j], U[i][j]);
    }
    if constexpr (C + 1 < NRE) eliminate<C + 1>(U, ip);
}

// The substep's increments x[n] of the partial densities from the concentrations
// sc [mol/cm3] (n < NRE) and their sum over all species
__device__ __forceinline__ void chem_increment(const double* sc, double mixture, double T, double dt, const DevParm& P,
                                               double* x) {
    double U[NRE][NRE + 1];
#pragma unroll
    for (int a = 0; a < NRE; ++a)
#pragma unroll
        for (int b = 0; b <= NRE; ++b) U[a][b] = a == b ? 1.0 : 0.0;
    const double lnT = log(T);
    const double invT = rcp_cubic(T);
    const double RsT = P.rs * T;
    const double iRsT = P.inv_rs * invT;
    double iE[NRE], z[NRE], inv[NRE];
    {
        const int h = T < 1000 ? 0 : 1;
#pragma unroll
        for (int n = 0; n < NRE; ++n) {
            inv[n] = rcp_cubic(sc[n] + 1e-20) * (dt * c_mder.inv_mw[n]);
            if (n < 2) {  // the elements: E = 1
                iE[n] = 1.0;
                z[n] = sc[n];
                continue;
            }
            const double* g = c_mder.gp[h][n - 2];
            const double t = fma(T, fma(T, fma(T, fma(T, g[4], g[3]), g[2]), g[1]), g[0]);
            const double ex = exp_tab(fma(g[5], invT, fma(g[6], lnT, t)));
            iE[n] = rcp_cubic(ex);
            z[n] = sc[n] * ex;
        }
    }
    const double alpha_a = fma(11.0, sc[2], fma(1.5, sc[0], mixture));
    // forward rate k = A T^b exp(-Ta/T), LiDryer.H:171-191
#define KF(A_, b_, Ta_) ((A_) * exp_tab(fma((b_), lnT, -(Ta_) * invT)))
#define KF0(A_, Ta_) ((A_) * exp_tab(-(Ta_) * invT))
#define ST(s0, s1, s2, s3, f0, f1, f2, f3, r0, r1, r2, r3) \
    Stoich { {s0, s1, s2, s3}, {f0, f1, f2, f3}, {r0, r1, r2, r3} }
    double k;
    // 0: H + O2 <=> O + OH
    k = KF(3.55e+15, -0.41, 8353.444256079512) * iE[3];
    rxn_accum(ST(3, 1, 4, 5, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[3] * z[1]), k * (z[4] * z[5]), inv, U);
    // 1: O + H2 <=> H + OH
    k = KF(50800.0, 2.67, 3165.2508657072367) * iE[4];
    rxn_accum(ST(4, 0, 3, 5, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[4] * z[0]), k * (z[3] * z[5]), inv, U);
    // 2: H2 + OH <=> H2O + H
    k = KF(2.16e+08, 1.51, 1726.0429999007667) * iE[5];
    rxn_accum(ST(0, 5, 2, 3, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[0] * z[5]), k * (z[2] * z[3]), inv, U);
    // 3: O + H2O <=> OH + OH
    k = KF(2.97e+06, 2.02, 6743.141748883461) * (iE[4] * iE[2]);
    rxn_accum(ST(4, 2, 5, -1, 1, 1, 0, 0, 0, 0, 2, 0), k * (z[4] * z[2]), k * (z[5] * z[5]), inv, U);
    // 4: H2 + M <=> H + H + M
    k = alpha_a * KF(4.58e+19, -1.4, 52526.05490660117);
    rxn_accum(ST(0, 3, -1, -1, 1, 0, 0, 0, 0, 2, 0, 0), k * z[0], k * RsT * (z[3] * z[3]), inv, U);
    // 5: O + O + M <=> O2 + M
    // (forward rate from the concentrations here and in 6: E_O^2 and E_O E_H leave
    // the range of doubles below about 85 K, where the products would be 0 x inf)
    k = alpha_a * (6.16e+15 * exp_tab(-0.5 * lnT));
    rxn_accum(ST(4, 1, -1, -1, 2, 0, 0, 0, 0, 1, 0, 0), k * (sc[4] * sc[4]), k * iRsT * (iE[4] * iE[4]) * z[1], inv, U);
    // 6: O + H + M <=> OH + M
    k = alpha_a * (4.71e+18 * invT);
    rxn_accum(ST(4, 3, 5, -1, 1, 1, 0, 0, 0, 0, 1, 0), k * (sc[4] * sc[3]), k * iRsT * (iE[4] * iE[3]) * z[5], inv, U);
    // 7: H + OH + M <=> H2O + M
    k = alpha_a * (3.8e+22 * (invT * invT)) * (iE[3] * iE[5]);
    rxn_accum(ST(3, 5, 2, -1, 1, 1, 0, 0, 0, 0, 1, 0), k * (z[3] * z[5]), k * iRsT * z[2], inv, U);
    // Troe falloff of the high-pressure rate khi with Fcent: the reduced pressure
    // redP = alpha klo / khi and its logarithm
    const auto falloff = [](double khi, double redP, double logPred, double logFcent) {
        const double troe_c = -0.4 - 0.67 * logFcent;
        const double troe_n = 0.75 - 1.27 * logFcent;
        const double xp = troe_c + logPred;
        const double troe = xp * rcp_cubic(fma(-0.14, xp, troe_n));
        const double F = exp_tab(2.302585092994046 * logFcent * rcp_cubic(fma(troe, troe, 1.0)));
        return khi * (redP * rcp_cubic(1.0 + redP)) * F;
    };
    const double log10e = 0.43429448190325182765;
    // 8: H + O2 (+M) <=> HO2 (+M), Fcent = 0.8
    {
        const double alpha = fma(-0.22, sc[1], fma(10.0, sc[2], mixture + sc[0]));
        const double a = fma(-2.32, lnT, -261.6741574193582 * invT);  // ln of T^-1.72 exp(-Ta / T) / T^0.6
        const double redP = alpha * (6.37e+20 / 1.48e+12) * exp_tab(a);
        const double logPred = log10e * ((log(alpha) + 19.880238125760414) + a);
        k = falloff(1.48e+12 * exp_tab(0.6 * lnT), redP, logPred, -0.09691001300805639) * iE[3];
    }
    rxn_accum(ST(3, 1, 6, -1, 1, 1, 0, 0, 0, 0, 1, 0), k * (z[3] * z[1]), k * iRsT * z[6], inv, U);
    const double i63 = iE[6] * iE[3], z63 = z[6] * z[3];
    // 9: HO2 + H <=> H2 + O2
    k = KF0(1.66e+13, 412.64001746898793) * i63;
    rxn_accum(ST(6, 3, 0, 1, 1, 1, 0, 0, 0, 0, 1, 1), k * z63, k * (z[0] * z[1]), inv, U);
    // 10: HO2 + H <=> OH + OH
    k = KF0(7.08e+13, 150.96586004962973) * i63;
    rxn_accum(ST(6, 3, 5, -1, 1, 1, 0, 0, 0, 0, 2, 0), k * z63, k * (z[5] * z[5]), inv, U);
    // 11: HO2 + O <=> O2 + OH
    k = 3.25e+13 * (iE[6] * iE[4]);
    rxn_accum(ST(6, 4, 1, 5, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[6] * z[4]), k * (z[1] * z[5]), inv, U);
    // 12: HO2 + OH <=> H2O + O2
    k = KF0(2.89e+13, -251.60976674938289) * (iE[6] * iE[5]);
    rxn_accum(ST(6, 5, 2, 1, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[6] * z[5]), k * (z[2] * z[1]), inv, U);
    // 13: HO2 + HO2 <=> H2O2 + O2 (two rate expressions, DUPLICATE)
    k = (KF0(4.2e+14, 6028.570011315214) + KF0(1.3e+11, -820.2478396029883)) * (iE[6] * iE[6]);
    rxn_accum(ST(6, 7, 1, -1, 2, 0, 0, 0, 0, 1, 1, 0), k * (z[6] * z[6]), k * (z[7] * z[1]), inv, U);
    // 14: H2O2 (+M) <=> OH + OH (+M), Troe falloff, Fcent = 0.5
    {
        const double a = (24355.825421340265 - 22846.166820843966) * invT;  // ln of exp(-Ta_lo / T) / exp(-Ta_hi / T)
        const double redP = alpha_a * (1.20e+17 / 2.95e+14) * exp_tab(a);
        const double logPred = log10e * ((log(alpha_a) + 6.008271665424363) + a);
        k = falloff(KF0(2.95e+14, 24355.825421340265), redP, logPred, -0.3010299956639812) * iE[7];
    }
    rxn_accum(ST(7, 5, -1, -1, 1, 0, 0, 0, 0, 2, 0, 0), k * z[7], k * RsT * (z[5] * z[5]), inv, U);
    const double i73 = iE[7] * iE[3], z73 = z[7] * z[3], e15 = exp_tab(-1997.7815479901 * invT);
    // 15: H2O2 + H <=> H2O + OH
    k = 2.41e+13 * e15 * i73;
    rxn_accum(ST(7, 3, 2, 5, 1, 1, 0, 0, 0, 0, 1, 1), k * z73, k * (z[2] * z[5]), inv, U);
    // 16: H2O2 + H <=> HO2 + H2
    k = KF0(4.82e+13, 4000.595291315188) * i73;
    rxn_accum(ST(7, 3, 6, 0, 1, 1, 0, 0, 0, 0, 1, 1), k * z73, k * (z[6] * z[0]), inv, U);
    // 17: H2O2 + O <=> OH + HO2
    k = 9.55e+06 * (T * T) * e15 * (iE[7] * iE[4]);
    rxn_accum(ST(7, 4, 5, 6, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[7] * z[4]), k * (z[5] * z[6]), inv, U);
    // 18: H2O2 + OH <=> HO2 + H2O (two rate expressions, DUPLICATE)
    k = (1.0e+12 + KF0(5.8e+14, 4810.778740248201)) * (iE[7] * iE[5]);
    rxn_accum(ST(7, 5, 6, 2, 1, 1, 0, 0, 0, 0, 1, 1), k * (z[7] * z[5]), k * (z[6] * z[2]), inv, U);
#undef KF
#undef KF0
#undef ST
    const double scale = 1e6 * dt;
#pragma unroll
    for (int n = 0; n < NRE; ++n) U[n][NRE] *= scale;
    // gauss, LiDryer.H:890-942: partial-pivot elimination, solution in x
    double ip[NRE];
    eliminate<0>(U, ip);
#pragma unroll
    for (int c = NRE - 1; c >= 0; --c) {
        double sum = U[c][NRE];
#pragma unroll
        for (int j = c + 1; j < NRE; ++j) sum = fma(-U[c][j], x[j], sum);
        x[c] = sum * ip[c];
    }
}

// ------------------------------------------------------------------ transport
__device__ __forceinline__ double poly5(double x, const double* c) {
    return fma(x, fma(x, fma(x, fma(x, c[4], c[3]), c[2]), c[1]), c[0]);
}

// mixtureProperties and getMixDiffCoeffsMass (ChemViscous.H:16-106) of one cell:
// Wilke viscosity, averaged conductivity and mixture-averaged diffusivities from the
// partial densities.  Bound by the FP64 pipe; the reference's expressions divide
// about 250 times per cell and take two square roots per species pair.  Here the
// pair constants are tables, each species and each binary diffusivity has one
// reciprocal, and each pair of the Wilke rule and of the diffusivities is visited
// once, adding to both its species' sums: 4977 -> 1158 FP64 instructions per cell,
// 685 -> 126 us on the 47430 cells around a 43x32x29 box, the FP64 pipe 87 % busy.
__device__ __forceinline__ void transport(double T, double p, double rho, const double* r, double& mu, double& lambda,
                                          double* D) {
    double X[NSP], yow = 0.0;
#pragma unroll
    for (int n = 0; n < NSP; ++n) {
        X[n] = r[n] * c_mder.inv_mw[n];
        yow += X[n];
    }
    const double iyow = rcp_cubic(yow);
#pragma unroll
    for (int n = 0; n < NSP; ++n) X[n] *= iyow;
    const double sqT = sqrt(T), logT = log(T), sqsqT = sqrt(sqT);
    double sq[NSP], isq[NSP], s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int k = 0; k < NSP; ++k) {
        sq[k] = sqsqT * poly5(logT, &c_mech.visc[k * 5]);
        isq[k] = rcp_cubic(sq[k]);
        const double lam = poly5(logT, &c_mech.cond[k * 5]);  // over sqrt(T)
        s1 = fma(X[k], lam, s1);
        s2 = fma(X[k], rcp_cubic(lam), s2);
    }
    lambda = 0.5 * sqT * (s1 + rcp_cubic(s2));
    // sum_j X_j phi_kj and sum_nn X_nn / D_(n nn), sum_nn X_nn W_nn / D_(n nn) of every
    // species (D over T^1.5)
    double ph[NSP], a1[NSP], a2[NSP], XW[NSP], W = 0.0;
#pragma unroll
    for (int k = 0; k < NSP; ++k) {
        ph[k] = X[k];
        a1[k] = a2[k] = 0.0;
        XW[k] = X[k] * c_mech.mw[k];
        W += XW[k];
    }
#pragma unroll
    for (int k = 1; k < NSP; ++k)
#pragma unroll
        for (int j = 0; j < k; ++j) {
            const double f = fma(sq[k] * isq[j], c_mder.wr14[k][j], 1.0);
            const double t = f * f * c_mder.wden[k][j];          // phi_kj
            const double v = sq[j] * isq[k];
            ph[k] = fma(X[j], t, ph[k]);
            ph[j] = fma(X[k], t * (v * v) * c_mder.wkj[k][j], ph[j]);  // phi_jk = phi_kj (mu_j / mu_k) (W_k / W_j)
            const int ic = j * NSP - (j * (j - 1)) / 2 + (k - j);     // upper-triangle index
            const double ib = rcp_cubic(poly5(logT, &c_mech.diff[ic * 5]));
            a1[k] = fma(X[j], ib, a1[k]);
            a1[j] = fma(X[k], ib, a1[j]);
            a2[k] = fma(XW[j], ib, a2[k]);
            a2[j] = fma(XW[k], ib, a2[j]);
        }
    double m = 0.0;
#pragma unroll
    for (int k = 0; k < NSP; ++k) m = fma(X[k] * (sq[k] * sq[k]), rcp_cubic(ph[k]), m);
    mu = m;
    const double pt = T * sqT * rcp_cubic(p);
#pragma unroll
    for (int n = 0; n < NSP; ++n) D[n] = pt * rcp_cubic(fma(a2[n], X[n] * rcp_cubic(W - XW[n]), a1[n]));
}

// ---- FP32 transport of the mixed form: the same fits and mixing rules with the
// species-pair constants of the Wilke rule precomputed in FP64 and rounded once
struct TransF {
    float visc[NSP * 5], cond[NSP * 5], diff[45 * 5];
    float mw[NSP];
    float wr14[NSP][NSP];   // (W_j / W_k)^(1/4)
    float den[NSP][NSP];    // 1 / sqrt(8 + 8 W_k / W_j)
    float wratio[NSP][NSP]; // W_j / W_k
};
__constant__ TransF c_trf;

__device__ __forceinline__ float dot5f(const float* x, const float* y) {
    return x[0] * y[0] + x[1] * y[1] + x[2] * y[2] + x[3] * y[3] + x[4] * y[4];
}

// mixtureProperties (ChemViscous.H:16-64) and getMixDiffCoeffsMass
// (ChemViscous.H:66-106) in FP32: mole fractions from the mass fractions,
// Wilke viscosity, averaged conductivity, mixture-averaged diffusivities
__device__ __forceinline__ void transport_f32(float T, float p, const float* Y, float& mu, float& lambda, float* D) {
    float X[NSP], tmp[NSP], yow = 0.0f;
#pragma unroll
    for (int i = 0; i < NSP; ++i) {
        tmp[i] = __fdividef(Y[i], c_trf.mw[i]);
        yow += tmp[i];
    }
    const float yowinv = __frcp_rn(yow);
#pragma unroll
    for (int i = 0; i < NSP; ++i) X[i] = tmp[i] * yowinv;
    const float sqT = sqrtf(T), logT = __logf(T), sqsqT = sqrtf(sqT);
    const float poly[5] = {1.0f, logT, logT * logT, logT * logT * logT, logT * logT * logT * logT};
    float mui[NSP], sqmui[NSP], lami[NSP];
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int k = 0; k < NSP; ++k) {
        sqmui[k] = sqsqT * dot5f(poly, &c_trf.visc[k * 5]);
        lami[k] = sqT * dot5f(poly, &c_trf.cond[k * 5]);
        mui[k] = sqmui[k] * sqmui[k];
        s1 += X[k] * lami[k];
        s2 += __fdividef(X[k], lami[k]);
    }
    lambda = 0.5f * (s1 + __frcp_rn(s2));
    float phi[NSP][NSP];
#pragma unroll
    for (int k = 0; k < NSP; ++k) {
#pragma unroll
        for (int j = 0; j < k; ++j) {
            const float f1 = 1.0f + __fdividef(sqmui[k], sqmui[j]) * c_trf.wr14[k][j];
            const float t = f1 * f1 * c_trf.den[k][j];
            phi[k][j] = t;
            phi[j][k] = __fdividef(t, __fdividef(mui[k], mui[j]) * c_trf.wratio[k][j]);
        }
        phi[k][k] = 1.0f;
    }
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < NSP; ++k) {
        float t = 0.0f;
#pragma unroll
        for (int j = 0; j < NSP; ++j) t += X[j] * phi[k][j];
        m += __fdividef(X[k] * mui[k], t);
    }
    mu = m;
    const float t32 = T * sqT;
    float mmw = 0.0f;
#pragma unroll
    for (int n = 0; n < NSP; ++n) mmw += X[n] * c_trf.mw[n];
#pragma unroll
    for (int n = 0; n < NSP; n++) {
        float a1 = 0.0f, a2 = 0.0f;
#pragma unroll
        for (int nn = 0; nn < NSP; nn++) {
            if (nn == n) continue;
            const int a = n < nn ? n : nn, b = n < nn ? nn : n;
            const int ic = a * NSP - (a * (a - 1)) / 2 + (b - a);
            const float bdinv = __frcp_rn(t32 * dot5f(poly, &c_trf.diff[ic * 5]));
            a1 += X[nn] * bdinv;
            a2 += X[nn] * c_trf.mw[nn] * bdinv;
        }
        a1 *= p;
        a2 *= __fdividef(p * X[n], mmw - c_trf.mw[n] * X[n]);
        D[n] = __frcp_rn(a1 + a2);
    }
}

}  // namespace ocfd
