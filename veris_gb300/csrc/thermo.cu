// Thermodynamics in float64: the surface-temperature Newton solve
// (veris/solve4temp.py:5-174) and ice growth with the ocean budgets
// (veris/growth.py:8-397).  Both are pointwise; one thread per padded point.
#include <cmath>

#include "stencil.cuh"
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
    // the adjoint's: qsub / qnum and aa1 ln10 of the saturation humidity, 1 / (iceConduct snowConduct)
    double qratio, aln10, rkk;
    double t2;            // Stanton number times friction velocity, density and heat capacity of the ocean
    double pFac[5];       // thickness of category l of five over the mean
    // solve4temp's saturation terms: qnum = bb1 cc0 and qsub = (1 - bb1) cc0, each as the sum of two
    // floats, and cc1
    float k0b_h, k0b_l;
    float odd_h[5], odd_l[5];   // 1 / (2l+1)
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
    for (int l = 0; l < 5; ++l) split(1.0 / (2 * l + 1), k.odd_h[l], k.odd_l[l]);
    k.t2 = p.stantonNr * p.uStarBase * p.rhoSea * p.cpWater;
    k.meltb = -k.t2 * (1 + (p.McPheeTaperFac - 1) / (1 + std::exp(-0.4 * (7 / 0.4)))) * k.qi;
    k.rhb = 1 / std::sqrt(p.hIce_reg);
    k.qratio = qsub / qnum;
    k.aln10 = 2663.5 * std::log(10.0);
    k.rkk = 1 / (p.iceConduct * p.snowConduct);
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
struct S4TCell {
    double lwc, Ta, d1ug, d1iug, slope, aI, aS, iceSW;
    double k0, e, e2;           // conductivity of the thinnest of five; exp(-1.5 hI[l]) of the next category, its step
    Ff k0f, d1u, d1i, Taf, aqh, TF;
    float Tin;
};

// what the adjoint reads of a category at its root: saturation humidity,
// conductivity, d absSW / d thickness (of the snow, or of the ice where there is none)
struct S4TRoot {
    double qs, k, dSW;
    bool up;
};

// what the categories share
template <int NC, bool BARE>
__device__ __forceinline__ S4TCell solve4temp_cell(const VerisParams &p, const GrowthK &gk, const S4TIn &x,
                                                   double Tin, double hI0, double hS0) {
    S4TCell c;
    c.lwc = dmax(p.minLWdown, x.LWdown);
    c.Ta = dmax(gk.TaMin, x.ATemp);
    const double ug = dmax(p.wSpeedMin, x.wSpeed);
    c.d1ug = p.s4t_d1 * ug;
    c.d1iug = p.s4t_d1i * ug;
    const bool wet = !gt64(gk.Twet, Tin) && !is_nan64(Tin), south = is_neg(x.fCori);
    c.aI = south ? (wet ? p.wetIceAlb_south : p.dryIceAlb_south) : (wet ? p.wetIceAlb : p.dryIceAlb);
    c.aS = south ? (wet ? p.wetSnowAlb_south : p.drySnowAlb_south) : (wet ? p.wetSnowAlb : p.drySnowAlb);
    c.slope = gk.rhCut * (c.aS - c.aI);
    c.iceSW = (1 - c.aI) * x.SWdown;   // absorbed and transmitted by snow-free ice
    // the five categories scale ice and snow thickness alike (veris/growth.py:62-71): hI[l] = (2l+1) hI[0]
    // and hS[l] = (2l+1) hS[0], so one conductivity and one exponential serve them all
    c.k0 = c.e = c.e2 = 0.0;
    if (BARE) {
        c.k0 = gk.k0b;
        c.k0f = Ff{gk.k0b_h, gk.k0b_l};
    } else if (NC == 5) {
        if (is_pos(hI0)) c.k0 = div_lane(p.iceConduct * p.snowConduct, fma(p.snowConduct, hI0, p.iceConduct * hS0));
        c.k0f = ff_of(c.k0);
        if (!is_pos(hS0)) {   // exp(-1.5 hI[l]) = exp(-1.5 hI[0])^(2l+1)
            c.e = exp_table(-1.5 * hI0);
            c.e2 = c.e * c.e;
        }
    }
    c.d1u = ff_of(c.d1ug);
    c.d1i = ff_of(c.d1iug);
    c.Taf = ff_of(c.Ta);
    c.aqh = ff_of(x.aqh);
    c.TF = ff_of(x.TempFrz);
    c.Tin = narrow(Tin);
    return c;
}

// category l, of ice thickness hI > 0 and snow thickness hS; T, Fio, Fia, pen
// as solve4temp returns them.  False where (BARE) a flux is not finite.
template <int NC, bool BARE>
__device__ __forceinline__ bool solve4temp_category(const VerisParams &p, const GrowthK &gk, const S4TIn &x,
                                                    S4TCell &c, int l, double hI, double hS, double &T, double &Fio,
                                                    double &Fia, double &oPen, S4TRoot *root = nullptr) {
    const bool snow = !BARE && is_pos(hS);
    const double emiss = snow ? p.snowEmiss : p.iceEmiss;
    double absSW = c.iceSW;
    oPen = 0.0;
    if (snow) {
        double alb = fma(hS, c.slope, c.aI);
        const bool deep = gt64(hS, p.hCut);
        if (deep) alb = c.aS;
        absSW = (1 - alb) * x.SWdown;
        if (root) root->dSW = deep ? 0.0 : -c.slope * x.SWdown;
    } else {
        if (NC != 5) c.e = exp_table(-1.5 * hI);
        const double pen = BARE ? gk.penb[l] : p.shortwave * c.e;
        if (!BARE && NC == 5) c.e *= c.e2;
        if (!BARE) oPen = -c.iceSW * pen;
        absSW = fma(-c.iceSW, pen, c.iceSW);
        if (root) root->dSW = 1.5 * c.iceSW * pen;
    }
    Ff k;
    double kd = 0.0;
    if (NC == 5) {
        k = ff_mul(c.k0f, Ff{gk.odd_h[l], gk.odd_l[l]});
    } else {
        kd = div_lane(p.iceConduct * p.snowConduct, fma(p.snowConduct, hI, p.iceConduct * hS));
        k = ff_of(kd);
    }
    const double lwabs = fma(-emiss, c.lwc, -absSW);
    const Ff lw = ff_of(lwabs), d3 = snow ? Ff{gk.d3s_h, gk.d3s_l} : Ff{gk.d3i_h, gk.d3i_l};
    const Ff qnum{gk.qn_h, gk.qn_l}, qsub{gk.qs_h, gk.qs_l};
    float t = c.Tin;
#pragma unroll 1
    for (int it = 0; it < 4; ++it) {
        const float rt = __frcp_rn(t), t2 = t * t;
        const float c3 = exp2f(8847.95548f * rt);
        const float D = c3 * 100000.f - gk.qs_h, rD = __frcp_rn(D);
        const float qs = gk.qn_h * rD;
        const float dqs = (gk.cc1 * c3 * rD) * rD * (rt * rt);
        const float R = k.h * (c.TF.h - t) -
                        (lw.h + t2 * t2 * d3.h + c.d1u.h * (t - c.Taf.h) + c.d1i.h * (qs - c.aqh.h));
        const float dF = 4.f * d3.h * t2 * t + c.d1u.h + c.d1i.h * dqs;
        t = fminf(fmaxf(t + R * __frcp_rn(k.h + dF), gk.Tmin_f), gk.Tmelt_f);
    }
    float dqs;
    const Ff qs = saturation_ff(t, qnum, qsub, gk.cc1, dqs);
    const float t2 = __fmul_rn(t, t);
    const Ff tt = ff_fast_sum(t2, fmaf(t, t, -t2));
    Ff Fc = ff_mul(k, ff_add(c.TF, -t));
    Ff Fa = ff_add(ff_mul(ff_mul(tt, tt), d3), lw);
    Fa = ff_add(Fa, ff_mul(c.d1u, ff_add(ff_neg(c.Taf), t)));
    Fa = ff_add(Fa, ff_mul(c.d1i, ff_add(qs, ff_neg(c.aqh))));
    const float res = (Fc.h - Fa.h) + (Fc.l - Fa.l);
    const float dF = 4.f * d3.h * t2 * t + c.d1u.h + c.d1i.h * dqs;
    const float step = res * __frcp_rn(k.h + dF);
    const float tn = fminf(fmaxf(t + step, gk.Tmin_f), gk.Tmelt_f);
    const double td = widen(t), Tmelt = p.celsius2K;
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
            Fa = ff_add(Fa, fmaf(6.f * d3.h * t2, d, dF) * d);
            const bool up = Fc.h > 0.f;
            const double F = ff_value(up ? Fc : Fa);
            Fio = up ? F : 0.0;
            Fia = up ? 0.0 : F;
            if (root) {
                root->up = up;
                root->k = ff_value(k);
                root->qs = ff_value(ff_add(qs, dqs * d));
            }
        }
        return true;
    }
    // veris/solve4temp.py:108-160: six iterations and the fluxes at their end
    const double qnumd = 0.622 * p.s4t_cc0, qsubd = (1.0 - 0.622) * p.s4t_cc0, d3d = emiss * p.stefBoltz;
    if (NC == 5) kd = c.k0 / (double)(2 * l + 1);
    double Fcd = 0.0, Fad = 0.0, qd = 0.0;
    T = td;
#pragma unroll 1
    for (int it = 0; it < 7; ++it) {
        const double rt = 1.0 / T, c3 = ::exp2(2663.5 * 3.32192809488736234787 * rt);
        const double s2 = T * T, D = c3 * 100000.0 - qsubd, q = qnumd / D;
        qd = q;
        Fcd = kd * (x.TempFrz - T);
        Fad = lwabs + s2 * s2 * d3d + c.d1ug * (T - c.Ta) + c.d1iug * (q - x.aqh);
        if (it == 6) break;
        const double Q = p.s4t_cc1 * c3 * (rt * rt) / (D * D);
        T = T + (Fcd - Fad) / (kd + 4 * d3d * (s2 * T) + c.d1ug + c.d1iug * Q);
        T = dmax(dmin(T, Tmelt), gk.Tmin);
    }
    const bool up = is_pos(Fcd);
    if (!BARE) {
        Fio = up ? Fcd : 0.0;
        Fia = up ? 0.0 : Fad;
        if (root) {
            root->up = up;
            root->k = kd;
            root->qs = qd;
        }
    }
    return finite64(up ? Fcd : Fad);
}

// the sums over the categories, hI (2l+1)/nITC and hS (2l+1)/nITC thick (veris/growth.py:62-92);
// NC = 5, or 1 for any other number.
// The loop stays rolled: unrolled it took 148 registers, 12 warps per SM, whose
// latency bound the kernel (float64 pipe 43 % busy, 448 us on 1440 x 720); rolled
// 317 us, and 265 with the kernel held to 80 registers, six CTAs per SM (four
// 286, five 269, eight 269).
template <int NC>
__device__ __forceinline__ void solve4temp_sums(const VerisParams &p, const GrowthK &gk, const S4TIn &x, double Tin,
                                                double hI, double hS, double &Tsum, double &Fio_sum, double &Fia_sum,
                                                double &pen_sum) {
    S4TCell c = solve4temp_cell<NC, false>(p, gk, x, Tin, hI * gk.pFac[0], hS * gk.pFac[0]);
    const int n = NC == 5 ? 5 : p.nITC;
#pragma unroll 1
    for (int l = 0; l < n; ++l) {
        double T = Tin, Fio = 0.0, Fia = 0.0, pen = 0.0;
        const double f = NC == 5 ? gk.pFac[l] : (double)(2 * l + 1) * p.recip_nITC;
        if (is_pos(hI) && is_pos(f))
            solve4temp_category<NC, false>(p, gk, x, c, l, hI * f, hS * f, T, Fio, Fia, pen);
        Tsum += T;
        Fio_sum += Fio;
        Fia_sum += Fia;
        pen_sum += pen;
    }
}

struct GrowthOut {
    double h, hs, A, TSurf, EmPmR, forc_salt, Qsw, Qnet, load, pen, rh;
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
__device__ __forceinline__ GrowthOut growth_point(const VerisParams &p, const GrowthK &gk, const Fields<double> &f, int64_t o,
                                                 double hIn, double hsIn, double AIn, double TSurfIn) {
    const double qi = gk.qi;
    const double qs = gk.qs;
    const bool noIce = is_zero(hIn) || is_zero(AIn);
    double h0 = hIn, hs0 = hsIn, A0 = AIn;
    if (noIce) {
        h0 = h0 * 0.0;
        hs0 = hs0 * 0.0;
        A0 = A0 * 0.0;
    }
    const bool isIce = is_pos(h0);
    const double rregA = rsqrt_lane(A0 * A0 + p.Area_reg);
    double hIa = isIce ? h0 * rregA : 0.0;
    const double rhIa = A0 * rsqrt_lane(h0 * h0 + p.hIce_reg);
    const double hSa = isIce ? hs0 * rregA : 0.0;
    hIa = dmax(hIa, 0.05);

    const double ocSalt = __ldg(f.ocSalt + o);
    const double TempFrz = p.tempFrz + p.dtempFrz_dS * ocSalt + p.celsius2K;
    S4TIn x;
    x.Tin = TSurfIn;
    x.TempFrz = TempFrz;
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = __ldg(f.fCori + o);
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);
    double Tsum = 0.0, Fio_sum = 0.0, Fia_sum = 0.0, pen_sum = 0.0;
    if (p.nITC == 5) solve4temp_sums<5>(p, gk, x, TSurfIn, hIa, hSa, Tsum, Fio_sum, Fia_sum, pen_sum);
    else solve4temp_sums<1>(p, gk, x, TSurfIn, hIa, hSa, Tsum, Fio_sum, Fia_sum, pen_sum);
    GrowthOut g;
    g.TSurf = Tsum * p.recip_nITC;
    const double An = A0 * p.recip_nITC;
    const double Fio = Fio_sum * An;
    double Fia = Fia_sum * An;
    const double pen = pen_sum * An;

    const double snowfall = __ldg(f.snowfall + o), precip = __ldg(f.precip + o);
    const bool cold = is_pos(A0) && mean_below(Tsum, gk.n, gk.rn, p.celsius2K);
    const double snowAcc = (cold ? snowfall + precip : snowfall) * p.rhoFresh2rhoSnow;
    const double rainToSea = cold ? 0.0 : precip;
    const double snowAccOverIce = snowAcc * A0 * p.deltatTherm;

    double gUnder = Fio * qi;
    if (is_zero(A0)) gUnder = 0.0;
    const double potMeltRate = -Fia * qs;
    const double potMelt = potMeltRate * p.deltatTherm;
    const bool allMelt = ge64(potMelt, hs0);
    const double meltRate = allMelt ? hs0 * p.recip_deltatTherm : potMeltRate;
    const double toSnow = allMelt ? -hs0 * p.recip_deltatTherm * gk.rqs : Fia;
    Fia = Fia - toSnow;
    const double gSurf = Fia * qi;
    const double gNet = (gUnder + gSurf) * rregA;

    const double t0 = 0.4, t1 = 7 / t0;
    const double t2 = gk.t2;
    const double sst = dmax(__ldg(f.theta + o), TempFrz);
    const double mltf = 1 + div_lane(p.McPheeTaperFac - 1, 1 + exp_table((A0 - t0) * t1));
    const double gML = -t2 * (sst - TempFrz) * mltf * qi;
    const double Qnet_in = __ldg(f.Qnet + o);
    const double gOW = qi * Qnet_in;

    const double dh = gNet * A0 + gOW * (1 - A0) + gML;
    const double dhs = (snowAcc - meltRate) * A0;
    const double half_rh = 0.5 * rhIa;
    double dA_oa = half_rh * gOW * (1 - A0);
    const bool grow = is_pos(gOW) && (is_pos(A0) || is_pos(dh));
    if (grow) dA_oa = gOW * (1 - A0);
    const double fC = __ldg(f.fCori + o);
    dA_oa = (grow && is_neg(fC)) ? dA_oa * p.recip_h0_south : dA_oa * p.recip_h0;
    const double dA_oi = !is_pos(gML) && !is_nan64(gML) ? half_rh * gML : 0.0;
    const double dA_ia = (!is_pos(gNet) && !is_nan64(gNet) && is_pos(h0)) ? half_rh * gNet * A0 : 0.0;
    const double dA = dA_oa + dA_oi + dA_ia;

    const double mask = __ldg(f.iceMask + o);
    const double mdt = mask * p.deltatTherm;
    double A = A0 + dA * mdt;
    double h = h0 + dh * mdt;
    double hs = hs0 + dhs * mdt;
    A = dmin(dmax(A, 0.0), 1.0);
    h = dmax(h, 0.0);
    hs = dmax(hs, 0.0);
    if (is_zero(h) || is_zero(A)) {
        A = A * 0.0;
        hs = hs * 0.0;
        h = h * 0.0;
    }
    const double hsub = (hs * p.rhoSnow + h * p.rhoIce) * p.recip_rhoSea;
    const double flood = dmax(0.0, hsub - h);
    h = h + flood;
    hs = hs - flood * p.rhoIce2rhoSnow;
    g.rh = rsqrt_lane(h * h + p.hIce_reg);
    g.h = h;
    g.hs = hs;
    g.A = A;

    g.Qsw = pen * A0 + __ldg(f.Qsw + o) * (1 - A0);
    const double dH = h - h0;
    const double melted = hs0 + snowAccOverIce - hs;
    const double E_ice = dH * gk.rqi;
    const double E_out = (A0 * (Fia + Fio + pen) + (1 - A0) * Qnet_in) * p.deltatTherm;
    g.Qnet = (E_out - E_ice) * p.recip_deltatTherm;
    double fw_ice = -dH * p.rhoIce2rhoFresh;
    if (p.saltIce_ref != 0.0 && is_pos(ocSalt) && gt64(ocSalt, p.saltIce_ref))
        fw_ice = fw_ice * (1 - p.saltIce_ref / ocSalt);
    const double salt_ref = dmin(p.saltIce_ref, ocSalt);
    const double osh = __ldg(f.os_hIceMean + o), oshs = __ldg(f.os_hSnowMean + o);
    double saltflux = 0.0;
    if (!is_zero(salt_ref)) saltflux = (dH + osh) * salt_ref * mask * p.rhoIce * p.recip_deltatTherm;
    const double fw_snow = melted * gk.rf2s;
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
                                            int64_t o, unsigned m, double TSurfIn, GrowthOut &g) {
    const double ocSalt = __ldg(f.ocSalt + o), fC = __ldg(f.fCori + o);
    S4TIn x;
    x.TempFrz = p.tempFrz + p.dtempFrz_dS * ocSalt + p.celsius2K;
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = fC;
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);
    S4TCell c = solve4temp_cell<5, true>(p, gk, x, TSurfIn, 0.0, 0.0);
    double Tsum = 0.0;
    bool finite = true;
#pragma unroll 1
    for (int l = 0; l < 5; ++l) {
        double T, unused0, unused1, unused2;
        finite = solve4temp_category<5, true>(p, gk, x, c, l, 0.0, 0.0, T, unused0, unused1, unused2) && finite;
        Tsum += T;
    }
    const double snowfall = __ldg(f.snowfall + o), precip = __ldg(f.precip + o);
    if (!__all_sync(m, finite && finite64(snowfall) && finite64(precip))) return false;
    g.TSurf = Tsum * p.recip_nITC;
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
__global__ void __launch_bounds__(128, 6) growth_kernel(VerisParams p, GrowthK gk, Fields<double> f, Dims d,
                                                     GrowthPtrs out, int i0, int i1) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = i0 + blockIdx.y * 4 + threadIdx.y;
    const unsigned m = __ballot_sync(0xffffffffu, i < i1 && j < d.NY);
    if (i >= i1 || j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    const double h0 = __ldg(f.hIceMean + o), hs0 = __ldg(f.hSnowMean + o), A0 = __ldg(f.Area + o);
    const double T0 = __ldg(f.TSurf + o);
    GrowthOut g;
    const bool water = p.nITC == 5 && (is_zero(h0) || is_zero(A0)) && finite64(h0) && finite64(hs0) && finite64(A0);
    if (!(__all_sync(m, water) && growth_bare(p, gk, f, o, m, T0, g)))
        g = growth_point(p, gk, f, o, h0, hs0, A0, T0);
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

// Adjoint of growth_point for the ice state (h, hs, A): given the adjoints of
// the new h, hs, A and TSurf, one forward pass for the values and one reverse
// pass (branches as in the forward).  TSurf enters Growth as the first guess
// of a converged iteration only: its adjoint is 0.
//
// solve4temp's categories: at the root T of R(T) = Fc(T) - Fia(T),
// dT = -R_theta / R_T with R_theta the residual's derivative at fixed T
// (through the conductivity k and the absorbed shortwave) and R_T =
// -(k + dFia/dT), the Newton iteration's own denominator; a root held by the
// melt or the minimum-temperature clamp has dT = 0.  (The converged Newton
// iterates have this derivative.)  Each category's shares in the adjoints of
// the ice and snow thickness are linear in the adjoints of the summed T, Fio
// and Fia, the last two known only after the sums, so the one loop collects
// the six coefficients (Q: through k, W: through the shortwave).
//
// 721 x 359 points: dual numbers for four inputs took 1.05 ms (1455 float64
// operations per point); this, with open water skipped, 0.23 ms (four CTAs per SM;
// six 0.24).
template <int NC>
__device__ __forceinline__ void growth_adjoint_point(const VerisParams &p, const GrowthK &gk,
                                                     const Fields<double> &f, int64_t o, double h0, double hs0,
                                                     double A0, double Tin, double l_h, double l_hs, double l_A,
                                                     double l_T, double &a_h, double &a_hs, double &a_A) {
    const bool isIce = is_pos(h0);
    const double rregA = rsqrt_lane(A0 * A0 + p.Area_reg), rregh = rsqrt_lane(h0 * h0 + p.hIce_reg);
    const double hIreg = isIce ? h0 * rregA : 0.0, hSa = isIce ? hs0 * rregA : 0.0;
    const bool thick = gt64(hIreg, 0.05);
    const double hIa = thick ? hIreg : 0.05;
    S4TIn x;
    x.TempFrz = p.tempFrz + p.dtempFrz_dS * __ldg(f.ocSalt + o) + p.celsius2K;
    x.LWdown = __ldg(f.LWdown + o);
    x.ATemp = __ldg(f.ATemp + o);
    x.wSpeed = __ldg(f.wSpeed + o);
    x.fCori = __ldg(f.fCori + o);
    x.SWdown = __ldg(f.SWdown + o);
    x.aqh = __ldg(f.aqh + o);

    // ---- the categories: sums, and the coefficients of their adjoints
    double Tsum = 0.0, Fio_sum = 0.0, Fia_sum = 0.0;
    double QT = 0.0, Qio = 0.0, Qia = 0.0, WT = 0.0, Wio = 0.0, Wia = 0.0;
    {
        S4TCell c = solve4temp_cell<NC, false>(p, gk, x, Tin, hIa * gk.pFac[0], hSa * gk.pFac[0]);
        const int n = NC == 5 ? 5 : p.nITC;
#pragma unroll 1
        for (int l = 0; l < n; ++l) {
            double T = Tin, Fio = 0.0, Fia = 0.0, pen;
            const double fl = NC == 5 ? gk.pFac[l] : (double)(2 * l + 1) * p.recip_nITC;
            if (is_pos(fl)) {
                S4TRoot r;
                solve4temp_category<NC, false>(p, gk, x, c, l, hIa * fl, hSa * fl, T, Fio, Fia, pen, &r);
                const double d3 = (is_pos(hSa * fl) ? p.snowEmiss : p.iceEmiss) * p.stefBoltz;
                const double T2 = T * T;
                // d qs / dT = qs (1 + qs qsub/qnum) aa1 ln10 / T^2
                const double dqs = r.qs * fma(r.qs, gk.qratio, 1.0) * (gk.aln10 * rcp_lane(T2));
                const double FiaT = fma(c.d1iug, dqs, fma(4.0 * d3, T2 * T, c.d1ug));
                const bool held = ge64(T, p.celsius2K) || ge64(gk.Tmin, T);
                const double s = held ? 0.0 : rcp_lane(r.k + FiaT);
                const double ks = r.k * s, fs = FiaT * s;
                const double u = r.k * r.k * fl * (x.TempFrz - T), w = r.dSW * fl;
                QT = fma(u, s, QT);
                WT = fma(w, s, WT);
                if (r.up) {
                    Qio = fma(u, held ? 1.0 : fs, Qio);
                    Wio = fma(-w, ks, Wio);
                } else {
                    Qia = fma(u, fs, Qia);
                    Wia = fma(-w, held ? 1.0 : ks, Wia);
                }
            }
            Tsum += T;
            Fio_sum += Fio;
            Fia_sum += Fia;
        }
    }

    // ---- forward (growth_point)
    const double An = A0 * p.recip_nITC, Fio = Fio_sum * An, Fia = Fia_sum * An;
    const bool cold = is_pos(A0) && mean_below(Tsum, gk.n, gk.rn, p.celsius2K);
    const double snowfall = __ldg(f.snowfall + o), precip = __ldg(f.precip + o);
    const double snowAcc = (cold ? snowfall + precip : snowfall) * p.rhoFresh2rhoSnow;
    const double potMeltRate = -Fia * gk.qs;
    const bool allMelt = ge64(potMeltRate * p.deltatTherm, hs0);
    const double meltRate = allMelt ? hs0 * p.recip_deltatTherm : potMeltRate;
    const double FiaR = allMelt ? Fia + hs0 * p.recip_deltatTherm * gk.rqs : 0.0;   // what melts ice
    const double G = ((is_zero(A0) ? 0.0 : Fio) + FiaR) * gk.qi;
    const double gNet = G * rregA;
    const double t0 = 0.4, t1 = 7 / t0;
    const double E = exp_table((A0 - t0) * t1), rE = rcp_lane(1.0 + E);
    const double M = p.McPheeTaperFac - 1;
    const double cML = -gk.t2 * (dmax(__ldg(f.theta + o), x.TempFrz) - x.TempFrz) * gk.qi;
    const double gML = cML * fma(M, rE, 1.0);
    const double gOW = gk.qi * __ldg(f.Qnet + o), open = 1.0 - A0;
    const double dh = gNet * A0 + gOW * open + gML;
    const double half = 0.5 * A0 * rregh;
    const bool grow = is_pos(gOW) && (is_pos(A0) || is_pos(dh));
    const double rh0 = (grow && is_neg(x.fCori)) ? p.recip_h0_south : p.recip_h0;
    const bool melts = !is_pos(gML) && !is_nan64(gML), thins = !is_pos(gNet) && !is_nan64(gNet) && isIce;
    const double dA_oa = (grow ? gOW : half * gOW) * open * rh0;
    const double dA = dA_oa + (melts ? half * gML : 0.0) + (thins ? half * gNet * A0 : 0.0);
    const double mdt = __ldg(f.iceMask + o) * p.deltatTherm;
    const double A1 = A0 + dA * mdt, h1 = h0 + dh * mdt, hs1 = hs0 + (snowAcc - meltRate) * A0 * mdt;
    const bool keepA = is_pos(A1) && gt64(1.0, A1), keeph = is_pos(h1), keephs = is_pos(hs1);

    // ---- reverse: flooding, the clips, the increments
    double gh = l_h, ghs = l_hs, gA = l_A;
    const double hc = keeph ? h1 : 0.0, hsc = keephs ? hs1 : 0.0;
    if (!gt64(0.0, (hsc * p.rhoSnow + hc * p.rhoIce) * p.recip_rhoSea - hc)) {
        const double gf = l_h - l_hs * p.rhoIce2rhoSnow;
        gh = fma(gf, p.rhoIce * p.recip_rhoSea - 1.0, gh);
        ghs = fma(gf, p.rhoSnow * p.recip_rhoSea, ghs);
    }
    if (!keeph || !is_pos(A1)) gh = ghs = gA = 0.0;   // no ice left
    if (!keephs) ghs = 0.0;
    if (!keepA) gA = 0.0;
    const double gdA = gA * mdt, gdh = gh * mdt, gdhs = ghs * mdt;
    const double g_melt = -gdhs * A0;
    double g_A = fma(gdhs, snowAcc - meltRate, gA);
    g_A = fma(gdh, gNet - gOW, g_A);
    double g_hs = ghs, g_h = gh;
    double g_gNet = gdh * A0, g_gML = gdh, g_half = 0.0;
    g_A = fma(-gdA * rh0, grow ? gOW : half * gOW, g_A);
    if (!grow) g_half = gdA * gOW * open * rh0;
    if (melts) {
        g_half = fma(gdA, gML, g_half);
        g_gML = fma(gdA, half, g_gML);
    }
    if (thins) {
        g_half = fma(gdA, gNet * A0, g_half);
        g_gNet = fma(gdA, half * A0, g_gNet);
        g_A = fma(gdA, half * gNet, g_A);
    }
    const double g_rhI = 0.5 * g_half * rregh;   // rhIa = A0 / sqrt(h0^2 + reg)
    g_A += g_rhI;
    g_h = fma(-g_rhI * A0 * h0, rregh * rregh, g_h);
    g_A = fma(-g_gML * cML * M * t1 * E, rE * rE, g_A);
    // ---- the fluxes
    const double g_G = g_gNet * rregA * gk.qi;   // per W/m2
    double g_rregA = g_gNet * G, g_Fio = is_zero(A0) ? 0.0 : g_G, g_Fia;
    if (allMelt) {
        g_Fia = g_G;
        g_hs = fma(fma(g_G, gk.rqs, g_melt), p.recip_deltatTherm, g_hs);
    } else {
        g_Fia = -gk.qs * g_melt;
    }
    g_A = fma(fma(g_Fio, Fio_sum, g_Fia * Fia_sum), p.recip_nITC, g_A);
    const double sT = l_T * p.recip_nITC, sio = g_Fio * An, sia = g_Fia * An;
    const double Q = -(QT * sT + Qio * sio + Qia * sia) * gk.rkk, W = WT * sT + Wio * sio + Wia * sia;
    double g_hI = Q * p.snowConduct, g_hS = Q * p.iceConduct;
    if (is_pos(hSa)) g_hS += W;
    else g_hI += W;
    if (!thick) g_hI = 0.0;
    if (isIce) {   // hIa = h0 rregA, hSa = hs0 rregA
        g_h = fma(g_hI, rregA, g_h);
        g_hs = fma(g_hS, rregA, g_hs);
        g_rregA = fma(g_hI, h0, fma(g_hS, hs0, g_rregA));
    }
    a_A = fma(-g_rregA * A0 * rregA, rregA * rregA, g_A);
    a_h = g_h;
    a_hs = g_hs;
}

__global__ void __launch_bounds__(128, 4) growth_adjoint_kernel(VerisParams p, GrowthK gk, Fields<double> f, Dims d,
                                                             const double *lh, const double *lhs, const double *lA,
                                                             const double *lT, double *oh, double *ohs, double *oA,
                                                             double *oT) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 4 + threadIdx.y;
    if (i >= d.NX || j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    const double h0 = __ldg(f.hIceMean + o), hs0 = __ldg(f.hSnowMean + o), A0 = __ldg(f.Area + o);
    const double l0 = lh[o], l1 = lhs[o], l2 = lA[o], l3 = lT[o];
    double a_h = 0.0, a_hs = 0.0, a_A = 0.0;
    if (is_zero(h0) || is_zero(A0)) {   // Growth multiplies the three by zero there
        a_h = (l0 + l1 + l2 + l3) * 0.0;
        a_hs = a_A = a_h;
    } else if (p.nITC == 5) {
        growth_adjoint_point<5>(p, gk, f, o, h0, hs0, A0, __ldg(f.TSurf + o), l0, l1, l2, l3, a_h, a_hs, a_A);
    } else {
        growth_adjoint_point<1>(p, gk, f, o, h0, hs0, A0, __ldg(f.TSurf + o), l0, l1, l2, l3, a_h, a_hs, a_A);
    }
    oh[o] = a_h;
    ohs[o] = a_hs;
    oA[o] = a_A;
    oT[o] = (l0 + l1 + l2 + l3) * 0.0;
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
