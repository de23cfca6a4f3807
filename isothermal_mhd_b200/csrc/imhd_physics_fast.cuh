// imhd_physics_fast.cuh -- FP32 evaluation of the Riemann fluxes and of the
// characteristic slope, on one interface or cell (F1) or on two at once (F2).
//
// Same mathematics as imhd_physics.cuh (which keeps the reference's
// operation order for the FP64 parity path), rearranged to issue fewer
// instructions:
//  * the states come as primitives and momenta, so that a velocity is divided
//    out once per cell and never again per face;
//  * divisions become one reciprocal and products, roots a reciprocal root;
//  * the jumps enter as dm - v drho, which both families of a pair share;
//  * the +/- eigenvector pairs of the fast, slow and Alfven families share
//    their terms: L.d is formed as P +/- Q, R.dm from the sums and
//    differences of the paired amplitudes;
//  * the continuity sign flips of the Roe eigenvectors (K98 eq. 2.20) are
//    dropped: they multiply both a left and the matching right eigenvector,
//    so they cancel in the dissipation term;
//  * the limiter is homogeneous, so the constant factors of the left
//    eigenvectors are applied once, after it;
//  * the eigenvector renormalisation constants come from forms without
//    cancellation: cs^2 = a^2 ca^2 / cf^2, the larger of cf^2 - ca^2 and
//    cf^2 - a^2 as a sum of positive terms and the smaller from their
//    product cf^2 bt^2.  Only near the triple point (cf^2 - cs^2 small) are
//    they evaluated in FP64 with the reference's limiting values.
#pragma once

#include "imhd_physics.cuh"
#include "imhd_value.cuh"

namespace imhd {

constexpr float kHalfRoot = 0.70710678118654752f;

// One side of an interface in the rotated frame: density, velocity (n, t1,
// t2), transverse field, momentum.
template <class V>
struct Side {
    V r, v[3], b[2], m[3];
};

// Flux components: rho, m_n, m_t1, m_t2, B_t1, B_t2 (the six of a sweep's
// flux fields, in their order).
//
// Roe flux of one interface (vanleer_mod.f90:2264-2863), FP32.
template <class V>
__device__ __forceinline__ void flux_roe_fast(const Side<V>& L, const Side<V>& R, V bn, float cs, float asqr, V* F,
                                              V& smax) {
    const V half = same<V>(0.5f), a1 = same<V>(cs), a2 = same<V>(asqr);
    const V sr = L.r + R.r, sx = L.v[0] + R.v[0], sy = L.v[1] + R.v[1], sz = L.v[2] + R.v[2];
    const V sb = L.b[0] + R.b[0], sc = L.b[1] + R.b[1];
    const V rho = half * sr, vx = half * sx, vy = half * sy, vz = half * sz;
    const V isr = vrsqrt(rho), srho = rho * isr, hisr = half * isr;
    const V qx = bn * isr, qy = sb * hisr, qz = sc * hisr;
    const V bt = fma(qy, qy, qz * qz), ca2 = qx * qx, dac = a2 - ca2, dd = dac - bt;
    const V t2 = vsqrt(fma(dd, dd, same<V>(4.0f * asqr) * bt));          // cf^2 - cs^2
    const V btt = bt + t2;
    const V cf2 = half * ((a2 + ca2) + btt), icf = vrsqrt(cf2), cf = cf2 * icf;
    const V ca = vabs(qx), css = (a1 * ca) * icf;                        // cf^2 cs^2 = a^2 ca^2
    smax = vmax2(smax, vabs(vx) + cf);

    // af = sqrt(cf^2 - ca^2) / sqrt(cf^2 - cs^2), as = sqrt(cf^2 - a^2) / sqrt(cf^2 - cs^2): the larger
    // radicand is big, the smaller cf^2 bt^2 / big; no transverse field: beta = (1, 1) / sqrt 2
    const V big = half * (vabs(dac) + btt), q = vrsqrt(big * t2);
    const V ib = each([](float b) { return b < 1.0e-30f ? 0.0f : rsqrtf(b); }, bt);
    const V cfbt = cf * (bt * ib);
    V af = vsel(dac, big, cfbt) * q, as = vsel(dac, cfbt, big) * q;
    if (any_less(t2, same<V>(1.0e-2f) * cf2)) {
#pragma unroll 1
        for (int l = 0; l < lanes_of<V>::n; ++l) {
            if (lane(t2, l) < 1.0e-2f * lane(cf2, l)) {
                double afd, asd;
                roe_alphas_fp64((double)lane(qx, l), (double)lane(qy, l), (double)lane(qz, l), (double)asqr, afd, asd);
                set_lane(af, l, (float)afd);
                set_lane(as, l, (float)asd);
            }
        }
    }
    const V gy = each([](float i, float g) { return i == 0.0f ? kHalfRoot : g; }, ib, qy * ib);
    const V gz = each([](float i, float g) { return i == 0.0f ? kHalfRoot : g; }, ib, qz * ib);
    const V ngy = same<V>(-1.0f) * gy;
    const V S = vsign(1.0f, qx);

    // characteristic amplitudes (K98 eq. 2.16-2.19, 2.27), the 1/2 of the flux average included
    const V d0 = R.r - L.r, nd0 = L.r - R.r;
    const V wn = fma(vx, nd0, R.m[0] - L.m[0]), w2 = fma(vy, nd0, R.m[1] - L.m[1]), w3 = fma(vz, nd0, R.m[2] - L.m[2]);
    const V e2 = R.b[0] - L.b[0], e3 = R.b[1] - L.b[1];
    const V wt = fma(gy, w2, gz * w3), wa = fma(gz, w2, ngy * w3);
    const V et = fma(gy, e2, gz * e3), ea = fma(gz, e2, ngy * e3);
    const V afc = af * a1, afcf = af * cf, asc = as * css, asca = as * ca, ascf = as * cf;
    const V quarter = same<V>(0.25f);
    const V i1 = quarter * vrcp(fma(afc, afc, ascf * ascf)), i2 = quarter * vrcp(fma(afc, afcf, asc * asca));
    const V X = srho * et, Sw = S * wt;
    const V Pf = i1 * fma(ascf, X, (afc * a1) * d0);
    const V Ps = i1 * ((ascf * cf) * d0 - afcf * X);
    const V Qf = i2 * (asc * Sw - afc * wn);
    const V Qs = i2 * fma(asca, wn, afcf * Sw);        // with the sign turned
    const V U = S * wa, W = srho * ea;                 // Alfven amplitudes without their 1/2 (in h below)

    // -|ev| c with Harten's entropy fix, delta = 0.3, on the fast and slow families
    // (vanleer_mod.f90:78, 2829-2833)
    auto harten = [](V ev, V c) {
        return each([](float e) {
                   const float a = -fabsf(e);
                   return a <= -0.3f ? a : __fmul_rn(__fadd_rn(a, -0.09f), 1.0f / 0.6f);
               }, ev) * c;
    };
    auto nabs = [](V ev) { return each([](float e) { return -fabsf(e); }, ev); };
    const V b0 = harten(vx - cf, Pf + Qf), b5 = harten(vx + cf, Pf - Qf);
    const V b2 = harten(vx - css, Ps - Qs), b3 = harten(vx + css, Ps + Qs);
    const V b1 = nabs(vx - ca) * (U + W), b4 = nabs(vx + ca) * (W - U);

    // minus sum_k beta_k R_k with the right eigenvectors of K98 eq. 2.12
    const V sF = b0 + b5, dF = b0 - b5, sS = b2 + b3, dS = b3 - b2, sA = b1 + b4, dA = b1 - b4;
    const V m = fma(af, sF, as * sS);
    const V q2 = S * fma(asca, dF, afc * dS);
    const V hA = (quarter * isr) * sA, SA = vsign(0.25f, qx) * dA;
    const V c4 = isr * (ascf * sF - (afc * (a1 * icf)) * sS);
    const V n1 = fma(vx, m, asc * dS - afcf * dF);
    const V n2 = fma(vy, m, fma(gy, q2, gz * SA)), n3 = fma(vz, m, fma(gz, q2, ngy * SA));
    const V n4 = fma(gy, c4, gz * hA), n5 = fma(gz, c4, ngy * hA);

    // plus the mean of the physical fluxes (vanleer_mod.f90:2765-2801)
    const V nb = same<V>(-1.0f) * bn;
    const V bb = fma(L.b[0], L.b[0], fma(L.b[1], L.b[1], fma(R.b[0], R.b[0], R.b[1] * R.b[1])));
    const V pr = fma(a2, sr, fma(half, bb, bn * nb));
    F[0] = fma(half, L.m[0] + R.m[0], m);
    F[1] = fma(half, fma(L.m[0], L.v[0], fma(R.m[0], R.v[0], pr)), n1);
    F[2] = fma(half, fma(L.m[0], L.v[1], fma(R.m[0], R.v[1], nb * sb)), n2);
    F[3] = fma(half, fma(L.m[0], L.v[2], fma(R.m[0], R.v[2], nb * sc)), n3);
    F[4] = fma(half, fma(L.v[0], L.b[0], fma(R.v[0], R.b[0], nb * sy)), n4);
    F[5] = fma(half, fma(L.v[0], L.b[1], fma(R.v[0], R.b[1], nb * sz)), n5);
}

// Fast magnetosonic speed given 1/rho, B_n^2 and the transverse field squared.
template <class V>
__device__ __forceinline__ V fast_speed_fast(V ir, V bn2, V bt2, float asqr) {
    const V bt = bt2 * ir, s = fma(bn2, ir, bt), a2 = same<V>(asqr), dd = a2 - s;
    const V t2 = vsqrt(fma(dd, dd, same<V>(4.0f * asqr) * bt));
    return vsqrt(same<V>(0.5f) * ((a2 + s) + t2));
}

// Signal speeds of HLLE and HLLD (vanleer_mod.f90:2895-2962, 3020-3086).
template <class V>
__device__ __forceinline__ void hll_speeds(const Side<V>& L, const Side<V>& R, V bn, float asqr, V& sL, V& sR, V& smax) {
    const V half = same<V>(0.5f), zero = same<V>(0.0f), bn2 = bn * bn;
    const V ia = vrcp(half * (L.r + R.r)), vxa = (half * (L.m[0] + R.m[0])) * ia;
    const V ab = half * (L.b[0] + R.b[0]), ac = half * (L.b[1] + R.b[1]);
    const V cL = fast_speed_fast(vrcp(L.r), bn2, fma(L.b[0], L.b[0], L.b[1] * L.b[1]), asqr);
    const V cR = fast_speed_fast(vrcp(R.r), bn2, fma(R.b[0], R.b[0], R.b[1] * R.b[1]), asqr);
    const V cm = fast_speed_fast(ia, bn2, fma(ab, ab, ac * ac), asqr);
    sL = vmin2(vmin2(L.v[0] - cL, vxa - cm), zero);
    sR = vmax2(vmax2(R.v[0] + cR, vxa + cm), zero);
    smax = vmax2(vmax2(smax, vabs(L.v[0]) + cL), vmax2(vabs(R.v[0]) + cR, vabs(vxa) + cm));
}

template <class V>
__device__ __forceinline__ void phys_flux_fast(const Side<V>& s, V bn, V nb, float asqr, V* F) {
    const V bt = fma(s.b[0], s.b[0], fma(s.b[1], s.b[1], bn * nb));
    F[0] = s.m[0];
    F[1] = fma(s.m[0], s.v[0], fma(same<V>(asqr), s.r, same<V>(0.5f) * bt));
    F[2] = fma(s.m[0], s.v[1], nb * s.b[0]);
    F[3] = fma(s.m[0], s.v[2], nb * s.b[1]);
    F[4] = fma(s.v[0], s.b[0], nb * s.v[1]);
    F[5] = fma(s.v[0], s.b[1], nb * s.v[2]);
}

// HLLE flux (vanleer_mod.f90:2867-2981), FP32.
template <class V>
__device__ __forceinline__ void flux_hlle_fast(const Side<V>& L, const Side<V>& R, V bn, float asqr, V* F, V& smax) {
    V sL, sR, FL[6], FR[6];
    hll_speeds(L, R, bn, asqr, sL, sR, smax);
    const V nb = same<V>(-1.0f) * bn;
    phys_flux_fast(L, bn, nb, asqr, FL);
    phys_flux_fast(R, bn, nb, asqr, FR);
    const V is = vrcp(sR - sL), x = sR * is, y = (same<V>(-1.0f) * sL) * is, z = sL * x;
    const V du[6] = {R.r - L.r, R.m[0] - L.m[0], R.m[1] - L.m[1], R.m[2] - L.m[2], R.b[0] - L.b[0], R.b[1] - L.b[1]};
#pragma unroll
    for (int c = 0; c < 6; ++c) F[c] = fma(x, FL[c], fma(y, FR[c], z * du[c]));
}

// Isothermal HLLD flux (Mignone 2007; vanleer_mod.f90:2986-3239), FP32.  Every
// star region is evaluated and the one of the interface selected; density and
// normal momentum take the HLL flux in all of them (F_K + s_K (U_hll - U_K)
// is the HLL flux), and the supersonic cases take the flux of one side.
template <class V>
__device__ __forceinline__ void flux_hlld_fast(const Side<V>& L, const Side<V>& R, V bn, float asqr, V* F, V& smax) {
    V sL, sR, FL[6], FR[6];
    hll_speeds(L, R, bn, asqr, sL, sR, smax);
    const V half = same<V>(0.5f), nb = same<V>(-1.0f) * bn, bn2 = bn * bn;
    phys_flux_fast(L, bn, nb, asqr, FL);
    phys_flux_fast(R, bn, nb, asqr, FR);
    const V is = vrcp(sR - sL), z = sR * sL;
    const V rs = ((sR * R.r - sL * L.r) - (FR[0] - FL[0])) * is;
    F[0] = fma(z, R.r - L.r, sR * FL[0] - sL * FR[0]) * is;
    F[1] = fma(z, R.m[0] - L.m[0], sR * FL[1] - sL * FR[1]) * is;
    const V irs = vrcp(rs), isr = vrsqrt(rs), vs = F[0] * irs, ax = vabs(bn) * isr;
    const V aL = vs - ax, aR = vs + ax;
    // star state of one side: m_t1, m_t2, B_t1, B_t2; the side's own where its
    // outer wave meets an Alfven wave
    auto star = [&](const Side<V>& u, V s, V* o) {
        const V xl = s - aL, xr = s - aR;
        const V i = vrcp(xl * xr), dv = s - u.v[0];
        const V t1 = (bn * (vs - u.v[0])) * i, t2 = ((u.r * dv) * dv - bn2) * (irs * i);
        const V near = vmin2(vabs(xl), vabs(xr)) - same<V>(1.0e-20f);
        o[0] = vsel(near, rs * u.v[1] - t1 * u.b[0], u.m[1]);
        o[1] = vsel(near, rs * u.v[2] - t1 * u.b[1], u.m[2]);
        o[2] = vsel(near, t2 * u.b[0], u.b[0]);
        o[3] = vsel(near, t2 * u.b[1], u.b[1]);
    };
    V uL[4], uR[4];
    star(L, sL, uL);
    star(R, sR, uR);
    const V srs = rs * isr, S = vsign(1.0f, bn), X = srs * S, iX = isr * S, nbi = nb * irs;
    const V naR = same<V>(-1.0f) * aR;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const V um = half * fma(X, uR[2 + c] - uL[2 + c], uL[c] + uR[c]);
        const V ub = half * fma(iX, uR[c] - uL[c], uL[2 + c] + uR[2 + c]);
        const V fm = fma(um, vs, nb * ub), fb = fma(vs, ub, um * nbi);
        F[2 + c] = vsel(aL, fma(sL, uL[c] - L.m[1 + c], FL[2 + c]),
                        vsel(naR, fma(sR, uR[c] - R.m[1 + c], FR[2 + c]), fm));
        F[4 + c] = vsel(aL, fma(sL, uL[2 + c] - L.b[c], FL[4 + c]),
                        vsel(naR, fma(sR, uR[2 + c] - R.b[c], FR[4 + c]), fb));
    }
    // sL = 0: everything leaves to the right; sR = 0: to the left
    if (any_less(vmin2(sR, same<V>(-1.0f) * sL), same<V>(1.0e-37f))) {
        const V nsR = same<V>(-1.0f) * sR;
#pragma unroll
        for (int c = 0; c < 6; ++c) F[c] = vsel(sL, FL[c], vsel(nsR, FR[c], F[c]));
    }
}

// Monotonised-central limiter times two, without its 1/2 and with the factor
// beta = 1.01 on the one-sided differences (mc_limit): the least of 2 beta dL,
// 2 beta dR and dL + dR where all are positive, the largest where all are
// negative, otherwise 0.
template <class V>
__device__ __forceinline__ V mc_twice(V dl, V dr) {
    const V k = same<V>((float)(2.0 * kMC_BETA));
    const V x = k * dl, y = k * dr, c = dl + dr;
    const V lo = vmin2(vmin2(x, y), c), hi = vmax2(vmax2(x, y), c);
    return each([](float a) { return fmaxf(a, 0.0f); }, lo) + each([](float a) { return fminf(a, 0.0f); }, hi);
}

// Limited characteristic slope of one cell (S08 A12/A22, vanleer_mod.f90:
// 941-1141, 1507-1546), FP32.  wm, w0, wp: rotated primitives of cells
// i-1, i, i+1; bn: face field at i+1/2.
template <bool PPM, class V>
__device__ __forceinline__ void plm_char_slope_fast(const V* wm, const V* w0, const V* wp, const V* wp2, V bn, float cs,
                                                    float asqr, V* delw) {
    const V half = same<V>(0.5f), a1 = same<V>(cs), a2 = same<V>(asqr);
    const V rho = w0[0], irs = vrsqrt(rho), rhos = rho * irs;
    const V bx = irs * bn, by = irs * w0[4], bz = irs * w0[5];
    const V bt = fma(by, by, bz * bz), ca2 = bx * bx, dac = a2 - ca2, dd = dac - bt;
    const V t2 = vsqrt(fma(dd, dd, same<V>(4.0f * asqr) * bt));          // cf^2 - cs^2
    const V btt = bt + t2;
    const V cf2 = half * ((a2 + ca2) + btt), icf = vrsqrt(cf2), cf = cf2 * icf;
    const V css = (a1 * vabs(bx)) * icf;                                 // cf^2 cs^2 = a^2 ca^2
    // af^2 = (a^2 - cs^2) / t2 = a^2 (cf^2 - ca^2) / (cf^2 t2), as^2 = (cf^2 - a^2) / t2; the larger of
    // cf^2 - ca^2 and cf^2 - a^2 is big, the smaller cf^2 bt^2 / big
    const V big = half * (vabs(dac) + btt), q = vrsqrt(big * t2);
    const V ib = each([](float b) { return b < 1.0e-30f ? 0.0f : rsqrtf(b); }, bt);
    const V sb = bt * ib;
    V af = (a1 * q) * vsel(dac, big * icf, sb), as = q * vsel(dac, cf * sb, big);
    if (any_less(t2, same<V>(1.0e-2f) * cf2)) {
#pragma unroll 1
        for (int l = 0; l < lanes_of<V>::n; ++l) {
            if (lane(t2, l) < 1.0e-2f * lane(cf2, l)) {
                double afd, asd;
                prim_alphas_fp64<float>((double)lane(rho, l), (double)lane(bn, l), (double)lane(w0[4], l),
                                        (double)lane(w0[5], l), (double)asqr, afd, asd);
                set_lane(af, l, (float)afd);
                set_lane(as, l, (float)asd);
            }
        }
    }
    const V gy = each([](float i, float g) { return i == 0.0f ? kHalfRoot : g; }, ib, by * ib);
    const V gz = each([](float i, float g) { return i == 0.0f ? kHalfRoot : g; }, ib, bz * ib);
    const V ngz = same<V>(-1.0f) * gz, naf = same<V>(-1.0f) * af;
    const V S = vsign(1.0f, bx);
    const V Cf = cf * af, Cs = css * as, Qf = Cf * S, Qs = Cs * S;
    const V k0 = (a2 * irs) * irs, k1 = a1 * irs, Si = S * irs;
    // left eigenvectors (S08 A22) times the differences, without the factors
    // 1/(2 a^2) (fast, slow) and 1/2 (Alfven)
    constexpr int NS = PPM ? 3 : 2;   // projected differences: w0-wm, wp-w0 (, wp2-wp)
    V aD[NS][6];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        V d[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) d[m] = s == 0 ? w0[m] - wm[m] : s == 1 ? wp[m] - w0[m] : wp2[m] - wp[m];
        V* a = aD[s];
        const V dvt = fma(gy, d[2], gz * d[3]), dbt = fma(gy, d[4], gz * d[5]);
        const V p0 = k0 * d[0], p1 = k1 * dbt;
        const V P = fma(af, p0, as * p1), Q = Qs * dvt - Cf * d[1];
        const V P2 = fma(as, p0, naf * p1), Q2 = fma(Cs, d[1], Qf * dvt);   // Q2 with the sign turned
        const V U = fma(gy, d[3], ngz * d[2]), W = Si * fma(gy, d[5], ngz * d[4]);
        a[0] = P + Q;
        a[5] = P - Q;
        a[2] = P2 - Q2;
        a[3] = P2 + Q2;
        a[1] = U + W;
        a[4] = W - U;
    }
    V dm[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        dm[k] = mc_twice(aD[0][k], aD[1][k]);
        if constexpr (PPM) dm[k] = mc_twice(aD[1][k], aD[2][k]) - dm[k];
    }
    // right eigenvectors (S08 A12) applied to the limited amplitudes, with the
    // factors left out above and the limiter's 1/2
    const V kN = same<V>(0.25f / asqr), kA = same<V>(0.25f);
    const V sf = kN * (dm[0] + dm[5]), df = kN * (dm[5] - dm[0]);
    const V ss = kN * (dm[2] + dm[3]), ds = kN * (dm[3] - dm[2]);
    const V sA = kA * (dm[1] + dm[4]), dA = kA * (dm[4] - dm[1]);
    const V tq = Qf * ds - Qs * df;
    const V ta = (a1 * rhos) * fma(as, sf, naf * ss);
    const V SA = (S * rhos) * sA;
    delw[0] = rho * fma(af, sf, as * ss);
    delw[1] = fma(Cf, df, Cs * ds);
    delw[2] = fma(gy, tq, gz * dA);
    delw[3] = gz * tq - gy * dA;
    delw[4] = fma(gy, ta, ngz * SA);
    delw[5] = fma(gz, ta, gy * SA);
}

// Primitive-variable slopes (prim_slope), FP32.
template <bool PPM, class V>
__device__ __forceinline__ void prim_slope_fast(const V* wm, const V* w0, const V* wp, const V* wp2, V* delw) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if constexpr (PPM)
            delw[k] = each([](float a, float b, float c) { return prim_ppm_limit(a, b, c); }, wm[k], w0[k], wp[k]) -
                      each([](float a, float b, float c) { return prim_ppm_limit(a, b, c); }, w0[k], wp[k], wp2[k]);
        else
            delw[k] = each([](float a, float b, float c) {
                const float dL = b - a, dR = c - b, dC = 0.5f * (dL + dR);
                return sgn1(dC) * vmin(vmin((float)kMC_BETA * fabsf(dL), (float)kMC_BETA * fabsf(dR)), fabsf(dC));
            }, wm[k], w0[k], wp[k]);
    }
}

template <int SOLVER, class V>
__device__ __forceinline__ void riemann_fast(const Side<V>& L, const Side<V>& R, V bn, float cs, float asqr, V* F,
                                             V& smax) {
    if constexpr (SOLVER == 1 || SOLVER == 4) flux_roe_fast(L, R, bn, cs, asqr, F, smax);   // 4: with protection fluxes
    else if constexpr (SOLVER == 2) flux_hlld_fast(L, R, bn, asqr, F, smax);
    else flux_hlle_fast(L, R, bn, asqr, F, smax);
}

// Slope of a sweep's reconstruction (scheme_recon: bit 0 PPM, bit 1 primitive
// variables): the characteristic slope or the primitive-variable one.
template <int RECON, class V>
__device__ __forceinline__ void recon_slope_fast(const V* wm, const V* w0, const V* wp, const V* wp2, V bn, float cs,
                                                 float asqr, V* delw) {
    constexpr bool PPM = (RECON & 1) != 0;
    if constexpr ((RECON & 2) != 0) prim_slope_fast<PPM>(wm, w0, wp, wp2, delw);
    else plm_char_slope_fast<PPM>(wm, w0, wp, wp2, bn, cs, asqr, delw);
}

// Interface side from a cell's primitives and a multiple h of its slope
// (+1/2: the state left of its upper face, -1/2: right of its lower one), or
// from a PPM edge.
template <class V>
__device__ __forceinline__ void side_of(const V* w, Side<V>& s) {
    s.r = w[0];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        s.v[m] = w[1 + m];
        s.m[m] = w[1 + m] * w[0];
    }
    s.b[0] = w[4];
    s.b[1] = w[5];
}
// PPM edge values (ppm_edges) of F1 values.
template <bool PRIM>
__device__ __forceinline__ void ppm_edges_fast(const F1* wm, const F1* w0, const F1* wp, const F1* dm, const F1* d0,
                                               F1* wl, F1* wr) {
    ppm_edges<float, PRIM>(&wm->v, &w0->v, &wp->v, &dm->v, &d0->v, &wl->v, &wr->v);
}
template <class V>
__device__ __forceinline__ void plm_side(const V* w, const V* d, float h, Side<V>& s) {
    V e[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) e[m] = fma(same<V>(h), d[m], w[m]);
    side_of(e, s);
}

}  // namespace imhd
