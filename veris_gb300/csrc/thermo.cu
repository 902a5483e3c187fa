// Thermodynamics in float64: the surface-temperature Newton solve
// (veris/solve4temp.py:5-174) and ice growth with the ocean budgets
// (veris/growth.py:8-397).  Both are pointwise; one thread per padded point.
#include <cmath>
#include <type_traits>

#include "stencil.cuh"
#include "dual.cuh"
#include "ffmath.cuh"

namespace veris {

struct S4TIn {
    double hI, hS, Tin, TempFrz;
    double LWdown, ATemp, wSpeed, fCori, SWdown, aqh;
};
struct S4TOut {
    double T, Fio, Fia, pen, fw;
};

__device__ __forceinline__ double dmax(double a, double b) { return gt64(a, b) ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return gt64(b, a) ? a : b; }

// veris/solve4temp.py:5-174 for one point
__device__ S4TOut solve4temp_point(const VerisParams &p, const S4TIn &x) {
    const double aa1 = 2663.5, aa2 = 12.537, bb1 = 0.622;
    const double Pa = 100000.0;
    const double one_m_bb1 = 1.0 - bb1;
    const double cc1 = p.s4t_cc1, cc2 = p.s4t_cc2, d1 = p.s4t_d1, d1i = p.s4t_d1i;
    const double Tmelt = p.celsius2K;
    const double SurfMeltTemp = Tmelt + p.wetAlbTemp;
    double T = x.Tin;
    const double lwc = dmax(p.minLWdown, x.LWdown);
    const double Ta = dmax(p.celsius2K + p.minTAir, x.ATemp);
    const double ug = dmax(p.wSpeedMin, x.wSpeed);
    const bool ice = x.hI > 0, snow = x.hS > 0;
    const double emiss = snow ? p.snowEmiss : p.iceEmiss;
    const double d3 = emiss * p.stefBoltz;
    const double lw = emiss * lwc;

    double aI = ice ? p.dryIceAlb : 0.0;
    double aS = ice ? p.drySnowAlb : 0.0;
    const bool wet = ice && T >= SurfMeltTemp;
    if (wet) { aI = p.wetIceAlb; aS = p.wetSnowAlb; }
    const bool south = ice && x.fCori < 0;
    if (south) { aI = p.dryIceAlb_south; aS = p.drySnowAlb_south; }
    if (south && T >= SurfMeltTemp) { aI = p.wetIceAlb_south; aS = p.wetSnowAlb_south; }
    double alb = ice ? aI + x.hS / p.hCut * (aS - aI) : 0.0;
    if (x.hS > p.hCut) alb = aS;
    if (x.hS == 0) alb = aI;

    double pen = ice ? p.shortwave * exp(-1.5 * x.hI) : 0.0;
    if (snow) pen = 0.0;
    const double penSW = ice ? -(1 - alb) * pen * x.SWdown : 0.0;
    const double absSW = ice ? (1 - alb) * (1 - pen) * x.SWdown : 0.0;
    const double k = ice ? p.iceConduct * p.snowConduct / (p.snowConduct * x.hI + p.iceConduct * x.hS) : 0.0;

    double Fc, Flh, Fia, dF;
    auto fluxes = [&](double t1) {
        const double t2 = t1 * t1, t3 = t2 * t1, t4 = t2 * t2;
        const double svp = pow(10.0, -aa1 / t1 + aa2);
        const double qs = ice ? bb1 * svp / (Pa - one_m_bb1 * svp) : 0.0;
        const double c3 = pow(10.0, aa1 / t1);
        const double den = cc2 - c3 * Pa;
        const double dqs = ice ? cc1 * c3 / (den * den * t2) : 0.0;
        Fc = ice ? k * (x.TempFrz - t1) : 0.0;
        Flh = ice ? d1i * ug * (qs - x.aqh) : 0.0;
        const double Flw = ice ? t4 * d3 : 0.0;
        const double Fs = ice ? d1 * ug * (t1 - Ta) : 0.0;
        Fia = ice ? (-lw - absSW + Flw + Fs + Flh) : 0.0;
        dF = ice ? 4 * d3 * t3 + d1 * ug + d1i * ug * dqs : 0.0;
    };
    for (int it = 0; it < 6; ++it) {
        fluxes(T);
        T = ice ? T + (Fc - Fia) / (k + dF) : 0.0;
        T = dmin(T, Tmelt);
        T = dmax(T, p.celsius2K + p.minTIce);
    }
    fluxes(T);
    S4TOut o;
    const bool up = Fc > 0;
    o.T = ice ? T : x.Tin;
    o.Fio = up ? Fc : 0.0;
    o.Fia = up ? 0.0 : Fia;
    o.pen = penSW;
    o.fw = ice ? Flh / p.lhSublim : 0.0;
    return o;
}

// step constants of Growth, formed once on the host (float64 divisions cost
// about ten fused multiply-adds each on GB300's float64 pipe)
struct GrowthK {
    double qi, qs;        // 1 / (rho lhFusion) of ice and snow
    double rqi, rqs;      // rho lhFusion of ice and snow
    double rf2s;          // 1 / rhoFresh2rhoSnow
    double rhCut;         // 1 / hCut
    double Tmin, Twet, TaMin;   // lowest ice temperature, start of wet albedos, lowest air temperature, in K
    double n, rn;         // nITC, 1 / nITC
    // open water: conductivity and penetrating fractions of the thinnest ice, the ocean's melting rate per K,
    // recip_hIceMean
    double k0b, penb[5], meltb, rhb;
    double t2;            // Stanton number times friction velocity, density and heat capacity of the ocean
    double pFac[5];       // thickness of category l of five over the mean
    // solve4temp's saturation terms: qnum = bb1 cc0 and qsub = (1 - bb1) cc0, each as the sum of two
    // floats, and cc1
    float k0b_h, k0b_l;
    float qn_h, qn_l, qs_h, qs_l, cc1;
    float d3s_h, d3s_l, d3i_h, d3i_l;   // emissivity times Stefan-Boltzmann over snow and ice
    float Tmin_f, Tmelt_f;
};

static GrowthK growth_k(const VerisParams &p) {
    GrowthK k;
    k.qi = 1 / (p.rhoIce * p.lhFusion);
    k.qs = 1 / (p.rhoSnow * p.lhFusion);
    k.rqi = p.rhoIce * p.lhFusion;
    k.rqs = p.rhoSnow * p.lhFusion;
    k.rf2s = 1 / p.rhoFresh2rhoSnow;
    k.rhCut = 1.0 / p.hCut;
    auto split = [](double x, float &h, float &l) {
        h = (float)x;
        l = (float)(x - (double)h);
    };
    split(p.snowEmiss * p.stefBoltz, k.d3s_h, k.d3s_l);
    split(p.iceEmiss * p.stefBoltz, k.d3i_h, k.d3i_l);
    k.Tmin = p.celsius2K + p.minTIce;
    k.Twet = p.celsius2K + p.wetAlbTemp;
    k.TaMin = p.celsius2K + p.minTAir;
    k.n = (double)p.nITC;
    k.rn = 1.0 / (double)p.nITC;
    for (int l = 0; l < 5; ++l) k.pFac[l] = (double)(2 * (l + 1) - 1) * p.recip_nITC;
    const double bb1 = 0.622, qnum = bb1 * p.s4t_cc0, qsub = (1.0 - bb1) * p.s4t_cc0;
    k.k0b = p.iceConduct * p.snowConduct / (p.snowConduct * (0.05 * k.pFac[0]));
    split(k.k0b, k.k0b_h, k.k0b_l);
    for (int l = 0; l < 5; ++l) k.penb[l] = p.shortwave * std::exp(-1.5 * (0.05 * k.pFac[l]));
    k.t2 = p.stantonNr * p.uStarBase * p.rhoSea * p.cpWater;
    k.meltb = -k.t2 * (1 + (p.McPheeTaperFac - 1) / (1 + std::exp(-0.4 * (7 / 0.4)))) * k.qi;
    k.rhb = 1 / std::sqrt(p.hIce_reg);
    split(qnum, k.qn_h, k.qn_l);
    split(qsub, k.qs_h, k.qs_l);
    k.cc1 = (float)p.s4t_cc1;
    k.Tmin_f = (float)k.Tmin;
    k.Tmelt_f = (float)p.celsius2K;
    return k;
}

// Saturation humidity over ice at the float temperature t, in double-float
// arithmetic (pairs of float32, ~2^-47): qs = bb1 svp / (Pa - (1-bb1) svp) =
// qnum / (10^(aa1/t) Pa - qsub) with svp = cc0 / 10^(aa1/t), as q0 + q1, and
// its derivative in float32.  10^(aa1/t) = 2^(A/t): with n the integer nearest
// A/t, A - n t is formed exactly (A in three parts), so the remainder
// f = (A - n t)/t carries no cancellation; 2^f = 2^(k/128) e^y with |y| <= 0.0028.
// A t outside the range of float arithmetic gives infinities or NaN here,
// which the caller's test of the step rejects.
__device__ __forceinline__ Ff saturation_ff(float t, Ff qnum, Ff qsub, float cc1, float &dqs) {
    constexpr float A_hi = 0x1.147fa4p+13f, A_mid = 0x1.a62a4p-12f, A_lo = -0x1.ffbd7ep-32f;   // 2663.5 log2(10)
    // products and sums whose rounding error is formed next must not be contracted
    const float r0 = __frcp_rn(t);
    const float n = rintf(A_hi * r0);
    const float nt = __fmul_rn(n, t);
    const float N0 = __fsub_rn(A_hi, nt), L0 = __fsub_rn(A_mid, fmaf(n, t, -nt));   // both exact
    const float N = __fadd_rn(N0, L0), L = __fsub_rn(L0, __fsub_rn(N, N0)) + A_lo;
    const float f0 = __fmul_rn(N, r0), f1 = (fmaf(-f0, t, N) + L) * r0;
    const float k = rintf(f0 * 128.f), g = fmaf(k, -0.0078125f, f0);
    constexpr float ln2_h = 0x1.62e43p-1f, ln2_l = -0x1.05c61p-29f;
    const float y = __fmul_rn(g, ln2_h);
    const float yl = fmaf(f1, ln2_h, fmaf(g, ln2_l, fmaf(g, ln2_h, -y)));
    const float y2 = __fmul_rn(y, y), y2l = fmaf(y, y, -y2) + 2.f * y * yl;
    const float c = y2 * y * fmaf(y, 1.f / 24.f, 1.f / 6.f);
    const float s = fmaf(0.5f, y2, y);   // e^y - 1 = s + sl
    const float sl = fmaf(0.5f, y2, __fsub_rn(y, s)) + (yl + fmaf(0.5f, y2l, c));
    const int ki = (int)k + 64;
    const float2 T = __ldg(EXP2_128F + min(max(ki, 0), 128));
    const float Ts = __fmul_rn(T.x, s);
    const float E = __fadd_rn(T.x, Ts);
    const float El = __fsub_rn(Ts, __fsub_rn(E, T.x)) + (fmaf(T.x, s, -Ts) + fmaf(T.x, sl, fmaf(T.y, s, T.y)));
    const float Pa = __uint_as_float(__float_as_uint(100000.f) + ((unsigned)min(max((int)n, -100), 100) << 23));
    const float X = __fmul_rn(E, Pa), Xl = fmaf(E, Pa, -X) + El * Pa;   // 10^(aa1/t) Pa
    const float D = __fsub_rn(X, qsub.h), Dl = __fsub_rn(__fsub_rn(X, D), qsub.h) + (Xl - qsub.l);
    const float rD = __frcp_rn(D);
    dqs = (cc1 * (X * 1e-5f) * rD) * rD * (r0 * r0);
    const float q = __fmul_rn(qnum.h, rD);
    return ff_fast_sum(q, (fmaf(-q, D, qnum.h) + fmaf(-q, Dl, qnum.l)) * rD);
}

// veris/solve4temp.py:5-174 for NC thickness categories of one cell in
// float64.  Bound by the float64 pipe, so what the results' last bits do not
// need runs elsewhere: eight float64 operations per category are left.
//
// Newton iterations in float32 bring T to ~1e-5 K of the root, at a float t.
// One more Newton step from t, with the residual Fc - Fia in double-float
// arithmetic (its error, ~1e-14 of the largest flux, is 1e-16 of T), ends the
// solve; the step d = (Fc - Fia) / (k + dF) itself needs float32 only.  The
// error left is below 1e-7 of d (float32 derivative) plus C d^2 with
// C = F''/2F' ~ 1e-3 / K, ~1e-10 K at the largest d accepted (4e-7 t, about
// 1e-4 K): far inside the parity of the fixed six iterations.  The fluxes at
// the new T are those at t plus their change over d: Fc's k d exactly, Fia's by
// its derivative (1e-7 of a change of at most 5e-3 W/m2) and the curvature of T^4.
// A category whose step is larger (or NaN) iterates in float64 from t, up to
// six times, with the six iterations' own formulas.
//
// BARE (NC = 5): open water, whose thinnest ice (0.05 m) without snow the
// reference solves for too: thicknesses and what depends on them alone are
// constants, and no fluxes are formed (the caller would multiply them by a
// zero concentration).  Returns false where a flux is not finite.
//
// 1440 x 720: with the residual's exponential and divisions in float64 and
// every comparison on its pipe (~80 operations per category) Growth took
// 1.66 ms; with the saturation term alone in double-float 0.65 ms; with the
// whole residual in it and the short form of open water (two thirds of a
// global grid's points) 0.45 ms.
template <int NC, bool BARE>
__device__ __forceinline__ bool solve4temp_f64(const VerisParams &p, const GrowthK &gk, const S4TIn &x, double Tin,
                                               const double *hI, const double *hS, double *oT, double *oFio,
                                               double *oFia, double *oPen) {
    const double Tmelt = p.celsius2K;
    const double lwc = dmax(p.minLWdown, x.LWdown);
    const double Ta = dmax(gk.TaMin, x.ATemp);
    const double ug = dmax(p.wSpeedMin, x.wSpeed);
    const double d1ug = p.s4t_d1 * ug, d1iug = p.s4t_d1i * ug;
    const bool wet = !gt64(gk.Twet, Tin) && !is_nan64(Tin), south = is_neg(x.fCori);
    const double aI = south ? (wet ? p.wetIceAlb_south : p.dryIceAlb_south) : (wet ? p.wetIceAlb : p.dryIceAlb);
    const double aS = south ? (wet ? p.wetSnowAlb_south : p.drySnowAlb_south) : (wet ? p.wetSnowAlb : p.drySnowAlb);
    const double slope = gk.rhCut * (aS - aI);
    const double iceSW = (1 - aI) * x.SWdown;   // absorbed and transmitted by snow-free ice
    // the five categories scale ice and snow thickness alike (veris/growth.py:62-71): hI[l] = (2l+1) hI[0]
    // and hS[l] = (2l+1) hS[0], so one conductivity and one exponential serve them all
    Ff k0{0.f, 0.f};
    double k0d = 0.0, e = 0.0, e2 = 0.0;
    bool finite = true;
    if (BARE) {
        k0d = gk.k0b;
        k0 = Ff{gk.k0b_h, gk.k0b_l};
    } else if (NC == 5) {
        if (is_pos(hI[0])) k0d = div_lane(p.iceConduct * p.snowConduct, fma(p.snowConduct, hI[0], p.iceConduct * hS[0]));
        k0 = ff_of(k0d);
        if (!is_pos(hS[0])) {   // exp(-1.5 hI[l]) = exp(-1.5 hI[0])^(2l+1)
            e = exp_table(-1.5 * hI[0]);
            e2 = e * e;
        }
    }
    const Ff d1u = ff_of(d1ug), d1i = ff_of(d1iug), Taf = ff_of(Ta), aqh = ff_of(x.aqh), TF = ff_of(x.TempFrz);
    const Ff qnum{gk.qn_h, gk.qn_l}, qsub{gk.qs_h, gk.qs_l};
    const float Tinf = narrow(Tin);
#pragma unroll
    for (int l = 0; l < NC; ++l) {
        const bool ice = BARE || is_pos(hI[NC == 5 ? 0 : l]), snow = !BARE && is_pos(hS[l]);
        if (!ice) {
            oT[l] = Tin;
            oFio[l] = oFia[l] = oPen[l] = 0.0;
            continue;
        }
        const double emiss = snow ? p.snowEmiss : p.iceEmiss;
        double absSW = iceSW;
        if (!BARE) oPen[l] = 0.0;
        if (snow) {
            double alb = fma(hS[l], slope, aI);
            if (gt64(hS[l], p.hCut)) alb = aS;
            absSW = (1 - alb) * x.SWdown;
        } else {
            if (NC != 5) e = exp_table(-1.5 * hI[l]);
            const double pen = BARE ? gk.penb[l] : p.shortwave * e;
            if (NC == 5) e *= e2;
            if (!BARE) oPen[l] = -iceSW * pen;
            absSW = fma(-iceSW, pen, iceSW);
        }
        Ff k;
        double kd = 0.0;
        if (NC == 5) {
            constexpr double inv_odd[5] = {1.0, 1.0 / 3.0, 1.0 / 5.0, 1.0 / 7.0, 1.0 / 9.0};
            const double q = inv_odd[l];   // a constant once unrolled
            k = ff_mul(k0, Ff{(float)q, (float)(q - (double)(float)q)});
        } else {
            kd = div_lane(p.iceConduct * p.snowConduct, fma(p.snowConduct, hI[l], p.iceConduct * hS[l]));
            k = ff_of(kd);
        }
        const double lwabs = fma(-emiss, lwc, -absSW);
        const Ff lw = ff_of(lwabs), d3 = snow ? Ff{gk.d3s_h, gk.d3s_l} : Ff{gk.d3i_h, gk.d3i_l};
        float t = Tinf;
        for (int it = 0; it < 4; ++it) {
            const float rt = __frcp_rn(t), t2 = t * t;
            const float c3 = exp2f(8847.95548f * rt);
            const float D = c3 * 100000.f - gk.qs_h, rD = __frcp_rn(D);
            const float qs = gk.qn_h * rD;
            const float dqs = (gk.cc1 * c3 * rD) * rD * (rt * rt);
            const float R = k.h * (TF.h - t) - (lw.h + t2 * t2 * d3.h + d1u.h * (t - Taf.h) + d1i.h * (qs - aqh.h));
            const float dF = 4.f * d3.h * t2 * t + d1u.h + d1i.h * dqs;
            t = fminf(fmaxf(t + R * __frcp_rn(k.h + dF), gk.Tmin_f), gk.Tmelt_f);
        }
        float dqs;
        const Ff qs = saturation_ff(t, qnum, qsub, gk.cc1, dqs);
        const float t2 = __fmul_rn(t, t);
        const Ff tt = ff_fast_sum(t2, fmaf(t, t, -t2));
        Ff Fc = ff_mul(k, ff_add(TF, -t));
        Ff Fia = ff_add(ff_mul(ff_mul(tt, tt), d3), lw);
        Fia = ff_add(Fia, ff_mul(d1u, ff_add(ff_neg(Taf), t)));
        Fia = ff_add(Fia, ff_mul(d1i, ff_add(qs, ff_neg(aqh))));
        const float res = (Fc.h - Fia.h) + (Fc.l - Fia.l);
        const float dF = 4.f * d3.h * t2 * t + d1u.h + d1i.h * dqs;
        const float step = res * __frcp_rn(k.h + dF);
        const float tn = fminf(fmaxf(t + step, gk.Tmin_f), gk.Tmelt_f);
        const double td = widen(t);
        double T;
        if (fabsf(tn - t) <= 4e-7f * t && fabsf(step) < 1e30f) {
            T = td + widen(step);
            float d = step;
            if (gt64(T, Tmelt)) {
                T = Tmelt;
                d = narrow(Tmelt - td);
            }
            if (gt64(gk.Tmin, T)) {
                T = gk.Tmin;
                d = narrow(gk.Tmin - td);
            }
            if (!BARE) {
                const float kd1 = __fmul_rn(k.h, d);
                Fc = ff_add(Fc, Ff{-kd1, -(fmaf(k.h, d, -kd1) + k.l * d)});
                Fia = ff_add(Fia, fmaf(6.f * d3.h * t2, d, dF) * d);
                const bool up = Fc.h > 0.f;
                const double F = ff_value(up ? Fc : Fia);
                oFio[l] = up ? F : 0.0;
                oFia[l] = up ? 0.0 : F;
            }
        } else {
            // veris/solve4temp.py:108-160: six iterations and the fluxes at their end
            const double qnumd = 0.622 * p.s4t_cc0, qsubd = (1.0 - 0.622) * p.s4t_cc0, d3d = emiss * p.stefBoltz;
            if (NC == 5) kd = k0d * (1.0 / (2 * l + 1));
            double Fcd = 0.0, Fiad = 0.0;
            T = td;
            for (int it = 0; it < 7; ++it) {
                const double rt = 1.0 / T, c3 = ::exp2(2663.5 * 3.32192809488736234787 * rt);
                const double s2 = T * T, D = c3 * 100000.0 - qsubd, q = qnumd / D;
                Fcd = kd * (x.TempFrz - T);
                Fiad = lwabs + s2 * s2 * d3d + d1ug * (T - Ta) + d1iug * (q - x.aqh);
                if (it == 6) break;
                const double Q = p.s4t_cc1 * c3 * (rt * rt) / (D * D);
                T = T + (Fcd - Fiad) / (kd + 4 * d3d * (s2 * T) + d1ug + d1iug * Q);
                T = dmax(dmin(T, Tmelt), gk.Tmin);
            }
            const bool up = is_pos(Fcd);
            if (!BARE) {
                oFio[l] = up ? Fcd : 0.0;
                oFia[l] = up ? 0.0 : Fiad;
            } else if (!finite64(up ? Fcd : Fiad)) {
                finite = false;
            }
        }
        oT[l] = T;
    }
    return finite;
}

// The same for dual numbers, when the adjoint needs the derivatives with
// respect to the ice state (branches follow the values).
template <int NC, class S>
__device__ void solve4temp_dual(const VerisParams &p, const GrowthK &gk, const S4TIn &x, const S &Tin, const S *hI, const S *hS,
                                S *oT, S *oFio, S *oFia, S *oPen) {
    const double aa1 = 2663.5, bb1 = 0.622, Pa = 100000.0;
    const double one_m_bb1 = 1.0 - bb1;
    const double cc0 = p.s4t_cc0, cc1 = p.s4t_cc1, cc2 = p.s4t_cc2, d1 = p.s4t_d1, d1i = p.s4t_d1i;
    const double Tmelt = p.celsius2K, Tmin = p.celsius2K + p.minTIce;
    const double SurfMeltTemp = Tmelt + p.wetAlbTemp;
    const double lwc = dmax(p.minLWdown, x.LWdown);
    const double Ta = dmax(p.celsius2K + p.minTAir, x.ATemp);
    const double ug = dmax(p.wSpeedMin, x.wSpeed);
    const double d1ug = d1 * ug, d1iug = d1i * ug;
    S k[NC], lwabs[NC];
    double d3[NC];
    bool ice[NC];
    // penetrating shortwave factor exp(-1.5 hI): the NC = 5 categories of one
    // cell have hI[l] = (2l+1) hI[0], so one exp and its odd powers serve all
    S e1[NC];
    if constexpr (NC == 5) {
        const S E = vexp(-1.5 * hI[0]), E2 = E * E;
        e1[0] = E;
#pragma unroll
        for (int l = 1; l < NC; ++l) e1[l] = e1[l - 1] * E2;
    } else {
#pragma unroll
        for (int l = 0; l < NC; ++l) e1[l] = vexp(-1.5 * hI[l]);
    }
    const double rhCut = gk.rhCut;
    // the categories scale ice and snow thickness alike (veris/growth.py:62-71):
    // with NC = 5, hI[l] = (2l+1) hI[0] and hS[l] = (2l+1) hS[0], so the
    // effective conductivity is k[0] / (2l+1): one division for the five
    S k0 = S(0.0);
    if constexpr (NC == 5)
        k0 = hI[0] > 0 ? p.iceConduct * p.snowConduct / (p.snowConduct * hI[0] + p.iceConduct * hS[0]) : S(0.0);
#pragma unroll
    for (int l = 0; l < NC; ++l) {
        ice[l] = hI[l] > 0;
        const bool snow = hS[l] > 0;
        const double emiss = snow ? p.snowEmiss : p.iceEmiss;
        d3[l] = emiss * p.stefBoltz;
        const double lw = emiss * lwc;
        double aI = ice[l] ? p.dryIceAlb : 0.0;
        double aS = ice[l] ? p.drySnowAlb : 0.0;
        if (ice[l] && Tin >= SurfMeltTemp) { aI = p.wetIceAlb; aS = p.wetSnowAlb; }
        const bool south = ice[l] && x.fCori < 0;
        if (south) { aI = p.dryIceAlb_south; aS = p.drySnowAlb_south; }
        if (south && Tin >= SurfMeltTemp) { aI = p.wetIceAlb_south; aS = p.wetSnowAlb_south; }
        S alb = ice[l] ? aI + hS[l] * rhCut * (aS - aI) : S(0.0);
        if (hS[l] > p.hCut) alb = S(aS);
        if (hS[l] == 0) alb = S(aI);
        S pen = ice[l] ? p.shortwave * e1[l] : S(0.0);
        if (snow) pen = S(0.0);
        oPen[l] = ice[l] ? -(1 - alb) * pen * x.SWdown : S(0.0);
        const S absSW = ice[l] ? (1 - alb) * (1 - pen) * x.SWdown : S(0.0);
        if constexpr (NC == 5) {
            constexpr double inv_odd[5] = {1.0, 1.0 / 3.0, 1.0 / 5.0, 1.0 / 7.0, 1.0 / 9.0};
            k[l] = ice[l] ? k0 * inv_odd[l] : S(0.0);
        } else {
            k[l] = ice[l] ? p.iceConduct * p.snowConduct / (p.snowConduct * hI[l] + p.iceConduct * hS[l]) : S(0.0);
        }
        lwabs[l] = -lw - absSW;
    }
    // Derivatives (dual numbers): implicit differentiation at the root.
    // The values come from the float64 solve itself (so every later
    // branch is taken as in the forward); at its root T* of
    // R(T) = Fc(T) - Fia(T), dT* = -R_theta / R_T with R_theta the
    // residual's derivative at fixed T (through the conductivity and
    // the absorbed radiation) and R_T = -(k + dFia/dT), the Newton
    // iteration's own denominator; a root held by the melt or the
    // minimum-temperature clamp has dT* = 0.  The converged Newton
    // iterates have this derivative (the Newton map's derivative in T
    // vanishes at the root), without iterating the dual numbers.
    double hIv[NC], hSv[NC], Tv[NC], Fiov[NC], Fiav[NC], Penv[NC];
#pragma unroll
    for (int l = 0; l < NC; ++l) {
        hIv[l] = val(hI[l]);
        hSv[l] = val(hS[l]);
    }
    solve4temp_f64<NC, false>(p, gk, x, val(Tin), hIv, hSv, Tv, Fiov, Fiav, Penv);
    const double aa1l2 = aa1 * 3.32192809488736234787;
    const double qnum = bb1 * cc0, qsub = one_m_bb1 * cc0;
#pragma unroll
    for (int l = 0; l < NC; ++l) {
        if (!ice[l]) {
            oT[l] = Tin;
            oFio[l] = S(0.0);
            oFia[l] = S(0.0);
            continue;
        }
        const double t = Tv[l], t3 = t * t * t;
        const double rt = 1.0 / t, c3 = ::exp2(aa1l2 * rt);
        const double qs = qnum / (c3 * Pa - qsub), den = cc2 - c3 * Pa;
        const double dqs = cc1 * c3 * (rt * rt) / (den * den);
        const double FiaT = 4 * d3[l] * t3 + d1ug + d1iug * dqs;
        const S Fc = k[l] * (x.TempFrz - t);
        const S Fia = lwabs[l] + (t3 * t * d3[l] + d1ug * (t - Ta) + d1iug * (qs - x.aqh));
        const bool held = t >= Tmelt || t <= Tmin;
        S dT = Fc - Fia;   // its derivative part: R_theta
        const double scale = held ? 0.0 : 1.0 / (val(k[l]) + FiaT);
        S T = Tin, Fo = Fc, Fa = Fia;
        T.v = t;
#pragma unroll
        for (int q = 0; q < (int)(sizeof(S::d) / sizeof(double)); ++q) {
            const double dTq = dT.d[q] * scale;
            T.d[q] = dTq;
            Fo.d[q] = Fc.d[q] - val(k[l]) * dTq;
            Fa.d[q] = Fia.d[q] + FiaT * dTq;
        }
        const bool up = Fiov[l] > 0;
        Fo.v = Fiov[l];
        Fa.v = Fiav[l];
        oT[l] = T;
        oFio[l] = up ? Fo : S(0.0);
        oFia[l] = up ? S(0.0) : Fa;
    }
}

template <int NC, class S>
__device__ __forceinline__ void solve4temp_multi(const VerisParams &p, const GrowthK &gk, const S4TIn &x,
                                                 const S &Tin, const S *hI, const S *hS, S *oT, S *oFio, S *oFia,
                                                 S *oPen) {
    if constexpr (std::is_same<S, double>::value) solve4temp_f64<NC, false>(p, gk, x, Tin, hI, hS, oT, oFio, oFia, oPen);
    else solve4temp_dual<NC, S>(p, gk, x, Tin, hI, hS, oT, oFio, oFia, oPen);
}

template <class S>
struct GrowthOut {
    S h, hs, A, TSurf, EmPmR, forc_salt, Qsw, Qnet, load, pen, rh;
};

// sum / n < limit as IEEE division has it (all categories at the melting point
// make the two sides equal): the division only where the product with the
// reciprocal is too near to tell
__device__ __forceinline__ bool mean_below(double sum, double n, double rn, double limit) {
    const double gap = sum * rn - limit;
    if (gt64(__hiloint2double(__double2hiint(gap) & 0x7fffffff, __double2loint(gap)), 1e-9)) return is_neg(gap);
    return sum / n < limit;
}

// veris/growth.py:8-397 for one point, from the ice state (h, hs, A, TSurf)
// and the forcing of point o
template <class S>
__device__ GrowthOut<S> growth_point(const VerisParams &p, const GrowthK &gk, const Fields<double> &f, int64_t o,
                                     S hIn, S hsIn, S AIn, S TSurfIn) {
    const double qi = gk.qi;
    const double qs = gk.qs;
    const bool noIce = vzero(hIn) || vzero(AIn);
    S h0 = hIn, hs0 = hsIn, A0 = AIn;
    if (noIce) {
        h0 = h0 * 0.0;
        hs0 = hs0 * 0.0;
        A0 = A0 * 0.0;
    }
    const bool isIce = vpos(h0);
    const S rregA = vrsqrt(A0 * A0 + p.Area_reg);
    S hIa = isIce ? h0 * rregA : S(0.0);
    const S rhIa = A0 * vrsqrt(h0 * h0 + p.hIce_reg);
    const S hSa = isIce ? hs0 * rregA : S(0.0);
    hIa = smax(hIa, S(0.05));

    const double ocSalt = __ldg(f.ocSalt + o);
    const double TempFrz = p.tempFrz + p.dtempFrz_dS * ocSalt + p.celsius2K;
    S4TIn x;
    x.Tin = val(TSurfIn);
    x.TempFrz = TempFrz;
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = __ldg(f.fCori + o);
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);
    S Tsum = 0, Fio_sum = 0, Fia_sum = 0, pen_sum = 0;
    if (p.nITC == 5) {
        S hIc[5], hSc[5], rT[5], rFio[5], rFia[5], rPen[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            hIc[l] = hIa * gk.pFac[l];
            hSc[l] = hSa * gk.pFac[l];
        }
        solve4temp_multi<5, S>(p, gk, x, TSurfIn, hIc, hSc, rT, rFio, rFia, rPen);
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            Tsum = Tsum + rT[l];
            Fio_sum = Fio_sum + rFio[l];
            Fia_sum = Fia_sum + rFia[l];
            pen_sum = pen_sum + rPen[l];
        }
    } else {
        for (int l = 0; l < p.nITC; ++l) {
            const double pFac = (double)(2 * (l + 1) - 1) * p.recip_nITC;
            S hIc[1] = {hIa * pFac}, hSc[1] = {hSa * pFac}, rT[1], rFio[1], rFia[1], rPen[1];
            solve4temp_multi<1, S>(p, gk, x, TSurfIn, hIc, hSc, rT, rFio, rFia, rPen);
            Tsum = Tsum + rT[0];
            Fio_sum = Fio_sum + rFio[0];
            Fia_sum = Fia_sum + rFia[0];
            pen_sum = pen_sum + rPen[0];
        }
    }
    GrowthOut<S> g;
    g.TSurf = Tsum * p.recip_nITC;
    const S An = A0 * p.recip_nITC;
    const S Fio = Fio_sum * An;
    S Fia = Fia_sum * An;
    const S pen = pen_sum * An;

    const double snowfall = __ldg(f.snowfall + o), precip = __ldg(f.precip + o);
    const bool cold = vpos(A0) && mean_below(val(Tsum), gk.n, gk.rn, p.celsius2K);
    const double snowAcc = (cold ? snowfall + precip : snowfall) * p.rhoFresh2rhoSnow;
    const double rainToSea = cold ? 0.0 : precip;
    const S snowAccOverIce = snowAcc * A0 * p.deltatTherm;

    S gUnder = Fio * qi;
    if (vzero(A0)) gUnder = S(0.0);
    const S potMeltRate = -Fia * qs;
    const S potMelt = potMeltRate * p.deltatTherm;
    const bool allMelt = vge(potMelt, hs0);
    const S meltRate = allMelt ? hs0 * p.recip_deltatTherm : potMeltRate;
    const S toSnow = allMelt ? -hs0 * p.recip_deltatTherm * gk.rqs : Fia;
    Fia = Fia - toSnow;
    const S gSurf = Fia * qi;
    const S gNet = (gUnder + gSurf) * rregA;

    const double t0 = 0.4, t1 = 7 / t0;
    const double t2 = gk.t2;
    const double sst = dmax(__ldg(f.theta + o), TempFrz);
    const S mltf = 1 + vdiv(p.McPheeTaperFac - 1, 1 + vexp((A0 - t0) * t1));
    const S gML = -t2 * (sst - TempFrz) * mltf * qi;
    const double Qnet_in = __ldg(f.Qnet + o);
    const double gOW = qi * Qnet_in;

    const S dh = gNet * A0 + gOW * (1 - A0) + gML;
    const S dhs = (snowAcc - meltRate) * A0;
    const S half_rh = 0.5 * rhIa;
    S dA_oa = half_rh * gOW * (1 - A0);
    const bool grow = is_pos(gOW) && (vpos(A0) || vpos(dh));
    if (grow) dA_oa = gOW * (1 - A0);
    const double fC = __ldg(f.fCori + o);
    dA_oa = (grow && is_neg(fC)) ? dA_oa * p.recip_h0_south : dA_oa * p.recip_h0;
    const S dA_oi = vle0(gML) ? half_rh * gML : S(0.0);
    const S dA_ia = (vle0(gNet) && vpos(h0)) ? half_rh * gNet * A0 : S(0.0);
    const S dA = dA_oa + dA_oi + dA_ia;

    const double mask = __ldg(f.iceMask + o);
    const double mdt = mask * p.deltatTherm;
    S A = A0 + dA * mdt;
    S h = h0 + dh * mdt;
    S hs = hs0 + dhs * mdt;
    A = smin(smax(A, S(0.0)), S(1.0));
    h = smax(h, S(0.0));
    hs = smax(hs, S(0.0));
    if (vzero(h) || vzero(A)) {
        A = A * 0.0;
        hs = hs * 0.0;
        h = h * 0.0;
    }
    const S hsub = (hs * p.rhoSnow + h * p.rhoIce) * p.recip_rhoSea;
    const S flood = smax(S(0.0), hsub - h);
    h = h + flood;
    hs = hs - flood * p.rhoIce2rhoSnow;
    g.rh = vrsqrt(h * h + p.hIce_reg);
    g.h = h;
    g.hs = hs;
    g.A = A;

    g.Qsw = pen * A0 + __ldg(f.Qsw + o) * (1 - A0);
    const S dH = h - h0;
    const S melted = hs0 + snowAccOverIce - hs;
    const S E_ice = dH * gk.rqi;
    const S E_out = (A0 * (Fia + Fio + pen) + (1 - A0) * Qnet_in) * p.deltatTherm;
    g.Qnet = (E_out - E_ice) * p.recip_deltatTherm;
    S fw_ice = -dH * p.rhoIce2rhoFresh;
    if (p.saltIce_ref != 0.0 && is_pos(ocSalt) && gt64(ocSalt, p.saltIce_ref))
        fw_ice = fw_ice * (1 - p.saltIce_ref / ocSalt);
    const double salt_ref = dmin(p.saltIce_ref, ocSalt);
    const double osh = __ldg(f.os_hIceMean + o), oshs = __ldg(f.os_hSnowMean + o);
    S saltflux = S(0.0);
    if (!is_zero(salt_ref)) saltflux = (dH + osh) * salt_ref * mask * p.rhoIce * p.recip_deltatTherm;
    const S fw_snow = melted * gk.rf2s;
    g.EmPmR = mask * ((-__ldg(f.evap + o) - precip) * (1 - A0) - rainToSea * A0 - __ldg(f.runoff + o) -
                      (fw_ice + fw_snow) * p.recip_deltatTherm) * p.rhoFresh +
              mask * (osh * p.rhoIce + oshs * p.rhoSnow) * p.recip_deltatTherm;
    g.forc_salt = g.EmPmR * ocSalt * p.recip_rhoFresh + saltflux;
    g.load = h * p.rhoIce + hs * p.rhoSnow;
    g.pen = pen;
    return g;
}

__global__ void solve4temp_kernel(VerisParams p, Fields<double> f, Dims d, const double *hI, const double *hS,
                                  const double *Tin, const double *TF, double *To, double *Fio, double *Fia,
                                  double *pen, double *fw) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 8 + threadIdx.y;
    if (i >= d.NX || j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    S4TIn x;
    x.hI = hI[o];
    x.hS = hS[o];
    x.Tin = Tin[o];
    x.TempFrz = TF[o];
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = __ldg(f.fCori + o);
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);
    const S4TOut r = solve4temp_point(p, x);
    To[o] = r.T;
    Fio[o] = r.Fio;
    Fia[o] = r.Fia;
    pen[o] = r.pen;
    fw[o] = r.fw;
}

struct GrowthPtrs {
    double *h, *hs, *A, *TSurf, *EmPmR, *forc_salt, *Qsw, *Qnet, *load, *pen, *rh;
};

// growth_point for a warp whose points (lanes of m) all are open water: no ice,
// snow or concentration, so that most of the terms vanish; about a fifth of the
// general point's float64 operations.  False where an input that the reference
// multiplies by zero is not finite (the caller takes the general point).
__device__ __forceinline__ bool growth_bare(const VerisParams &p, const GrowthK &gk, const Fields<double> &f,
                                            int64_t o, unsigned m, double TSurfIn, GrowthOut<double> &g) {
    const double ocSalt = __ldg(f.ocSalt + o), fC = __ldg(f.fCori + o);
    S4TIn x;
    x.TempFrz = p.tempFrz + p.dtempFrz_dS * ocSalt + p.celsius2K;
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = fC;
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);
    const double none[1] = {0.0};
    double T[5];
    const bool finite = solve4temp_f64<5, true>(p, gk, x, TSurfIn, none, none, T, nullptr, nullptr, nullptr);
    const double snowfall = __ldg(f.snowfall + o), precip = __ldg(f.precip + o);
    if (!__all_sync(m, finite && finite64(snowfall) && finite64(precip))) return false;
    g.TSurf = ((((T[0] + T[1]) + T[2]) + T[3]) + T[4]) * p.recip_nITC;
    const double Qnet = __ldg(f.Qnet + o), mask = __ldg(f.iceMask + o);
    const double gOW = gk.qi * Qnet;
    const double dh = gOW + gk.meltb * (dmax(__ldg(f.theta + o), x.TempFrz) - x.TempFrz);
    const double mdt = mask * p.deltatTherm;
    double h = dmax(dh * mdt, 0.0), A = 0.0;
    if (is_pos(gOW) && is_pos(dh))
        A = dmin(dmax(gOW * (is_neg(fC) ? p.recip_h0_south : p.recip_h0) * mdt, 0.0), 1.0);
    const bool some = !is_zero(h) && !is_zero(A);
    const double osh = __ldg(f.os_hIceMean + o), oshs = __ldg(f.os_hSnowMean + o);
    g.h = g.hs = g.A = g.load = g.pen = 0.0;
    g.rh = gk.rhb;
    g.Qsw = __ldg(f.Qsw + o);
    double E = Qnet * p.deltatTherm, dry = -__ldg(f.evap + o) - precip - __ldg(f.runoff + o);
    if (__any_sync(m, some)) {   // new ice
        h = some ? h : 0.0;
        const double flood = dmax(0.0, h * p.rhoIce * p.recip_rhoSea - h);
        h = h + flood;
        const double hs = -flood * p.rhoIce2rhoSnow;
        g.A = some ? A : 0.0;
        g.h = h;
        g.hs = hs;
        g.rh = rsqrt_lane(fma(h, h, p.hIce_reg));
        E -= h * gk.rqi;
        double fw = -h * p.rhoIce2rhoFresh;
        if (p.saltIce_ref != 0.0 && is_pos(ocSalt) && gt64(ocSalt, p.saltIce_ref)) fw *= 1 - p.saltIce_ref / ocSalt;
        dry -= (fw - hs * gk.rf2s) * p.recip_deltatTherm;
        g.load = h * p.rhoIce + hs * p.rhoSnow;
    }
    g.Qnet = E * p.recip_deltatTherm;
    double emp = mask * dry * p.rhoFresh;
    if (__any_sync(m, !is_zero(osh) || !is_zero(oshs)))
        emp += mask * (osh * p.rhoIce + oshs * p.rhoSnow) * p.recip_deltatTherm;
    g.EmPmR = emp;
    double salt = emp * ocSalt * p.recip_rhoFresh;
    const double salt_ref = dmin(p.saltIce_ref, ocSalt);
    if (!is_zero(salt_ref)) salt += (g.h + osh) * salt_ref * mask * p.rhoIce * p.recip_deltatTherm;
    g.forc_salt = salt;
    return true;
}

// rows [i0, i1) of the padded array (Growth is pointwise)
__global__ void __launch_bounds__(128) growth_kernel(VerisParams p, GrowthK gk, Fields<double> f, Dims d,
                                                     GrowthPtrs out, int i0, int i1) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = i0 + blockIdx.y * 4 + threadIdx.y;
    const unsigned m = __ballot_sync(0xffffffffu, i < i1 && j < d.NY);
    if (i >= i1 || j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    const double h0 = __ldg(f.hIceMean + o), hs0 = __ldg(f.hSnowMean + o), A0 = __ldg(f.Area + o);
    const double T0 = __ldg(f.TSurf + o);
    GrowthOut<double> g;
    const bool water = p.nITC == 5 && (is_zero(h0) || is_zero(A0)) && finite64(h0) && finite64(hs0) && finite64(A0);
    if (!(__all_sync(m, water) && growth_bare(p, gk, f, o, m, T0, g)))
        g = growth_point<double>(p, gk, f, o, h0, hs0, A0, T0);
    out.h[o] = g.h;
    out.hs[o] = g.hs;
    out.A[o] = g.A;
    out.TSurf[o] = g.TSurf;
    out.EmPmR[o] = g.EmPmR;
    out.forc_salt[o] = g.forc_salt;
    out.Qsw[o] = g.Qsw;
    out.Qnet[o] = g.Qnet;
    out.load[o] = g.load;
    out.pen[o] = g.pen;
    out.rh[o] = g.rh;
}

// adjoint of growth for the ice state: l_in = J^T l_out over (h, hs, A, TSurf)
__global__ void __launch_bounds__(128) growth_adjoint_kernel(VerisParams p, GrowthK gk, Fields<double> f, Dims d,
                                                             const double *lh, const double *lhs, const double *lA,
                                                             const double *lT, double *oh, double *ohs, double *oA,
                                                             double *oT) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 4 + threadIdx.y;
    if (i >= d.NX || j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    using D = Dual<4>;
    const GrowthOut<D> g = growth_point<D>(p, gk, f, o, D::var(f.hIceMean[o], 0), D::var(f.hSnowMean[o], 1),
                                           D::var(f.Area[o], 2), D::var(f.TSurf[o], 3));
    const double l0 = lh[o], l1 = lhs[o], l2 = lA[o], l3 = lT[o];
    double r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = l0 * g.h.d[k] + l1 * g.hs.d[k] + l2 * g.A.d[k] + l3 * g.TSurf.d[k];
    oh[o] = r[0];
    ohs[o] = r[1];
    oA[o] = r[2];
    oT[o] = r[3];
}

}  // namespace veris

using namespace veris;

extern "C" {

int veris_solve4temp_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs,
                         const double *hI, const double *hS, const double *Tin, const double *TF, double *To,
                         double *Fio, double *Fia, double *pen, double *fw, veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && hI && hS && Tin && TF && To && Fio && Fia && pen && fw, VERIS_ERR_ARG);
    dim3 gr((d.NY + 31) / 32, (d.NX + 7) / 8);
    solve4temp_kernel<<<gr, dim3(32, 8), 0, (cudaStream_t)s>>>(
        *p, *reinterpret_cast<const Fields<double> *>(vs), d, hI, hS, Tin, TF, To, Fio, Fia, pen, fw);
    return launch_status();
}

int veris_growth_adjoint_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, const double *lh,
                             const double *lhs, const double *lA, const double *lT, double *oh, double *ohs,
                             double *oA, double *oT, veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && lh && lhs && lA && lT && oh && ohs && oA && oT, VERIS_ERR_ARG);
    VERIS_REQUIRE(p->nITC >= 1 && p->nITC <= 64, VERIS_ERR_ARG);
    dim3 gr((d.NY + 31) / 32, (d.NX + 3) / 4);
    growth_adjoint_kernel<<<gr, dim3(32, 4), 0, (cudaStream_t)s>>>(*p, growth_k(*p), *reinterpret_cast<const Fields<double> *>(vs),
                                                                   d, lh, lhs, lA, lT, oh, ohs, oA, oT);
    return launch_status();
}

int veris_growth_rows_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, double *h,
                          double *hs, double *A, double *TSurf, double *EmPmR, double *forc_salt, double *Qsw,
                          double *Qnet, double *load, double *pen, double *rh, int32_t row_begin, int32_t row_end,
                          veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && h && hs && A && TSurf && EmPmR && forc_salt && Qsw && Qnet && load && pen && rh,
                  VERIS_ERR_ARG);
    VERIS_REQUIRE(p->nITC >= 1 && p->nITC <= 64, VERIS_ERR_ARG);
    VERIS_REQUIRE(row_begin >= 0 && row_begin < row_end && row_end <= d.NX, VERIS_ERR_ARG);
    GrowthPtrs out{h, hs, A, TSurf, EmPmR, forc_salt, Qsw, Qnet, load, pen, rh};
    dim3 gr((d.NY + 31) / 32, (row_end - row_begin + 3) / 4);
    growth_kernel<<<gr, dim3(32, 4), 0, (cudaStream_t)s>>>(*p, growth_k(*p), *reinterpret_cast<const Fields<double> *>(vs), d,
                                                            out, row_begin, row_end);
    return launch_status();
}

int veris_growth_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, double *h,
                     double *hs, double *A, double *TSurf, double *EmPmR, double *forc_salt, double *Qsw,
                     double *Qnet, double *load, double *pen, double *rh, veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    return veris_growth_rows_f64(g, p, vs, h, hs, A, TSurf, EmPmR, forc_salt, Qsw, Qnet, load, pen, rh, 0, d.NX,
                                 s);
}

}  // extern "C"
