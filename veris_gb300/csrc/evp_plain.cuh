// The mEVP subcycle on one tile, plain form (veris/evp_solver.py:21-254):
// every option, any masks and metrics, the reference's order of operations.
// Used by the plain loop (evp.cu) and, on states that the folded float64 form
// does not cover, by the drop-in's loop (evp_auto64.cu).
//
// A CTA owns at most TI rows by 32 columns of padded points (x rows by y
// columns, y contiguous).  It recomputes the intermediates it needs on a thin
// ring around them into shared memory, so one launch does the whole subcycle:
//
//   A  e12 (and rAz*e12^2) at Z points  [-1, ti+1] x [-1, TJ+1]
//   B  e11, e22, Delta, zeta, press at C [-1, ti] x [-1, TJ]; on [-1, ti) x
//      [-1, TJ) also the new sigma1/sigma2, sig11/sig22, the drag
//      coefficients and the Coriolis terms at C
//   C  zeta at Z and the new sigma12      [0, ti] x [0, TJ]
//   D  stress divergence, forcing, implicit drag and the new u, v on the tile
//
// The new u, v are stored together with their periodic images in the halo
// columns (and rows) that the reference's fill_overlap_uv refreshes
// (veris/evp_solver.py:190).  Stresses are not halo-filled, as in the
// reference.
#pragma once

#include "stencil.cuh"

namespace veris {

constexpr int EVP_THREADS = 256;

template <class T>
struct EvpIO {
    const T *u, *v, *s1, *s2, *s12;   // state at the start of the subcycle
    T *uo, *vo, *s1o, *s2o, *s12o;    // state at its end
    const T *uNm1, *vNm1;             // velocities of the previous time step
    T *aCo = nullptr;                 // adaptive EVP: alphaC of the subcycle, when not null
};

// shared memory of a tile of at most TI rows x 32 columns
template <class T, int TI, bool ADAPT, bool SIDE, bool BASAL>
struct PlainSmem {
    static constexpr int TJ = 32;
    // widths of the regions
    static constexpr int WZ = TJ + 3, HZ = TI + 3;   // stage A
    static constexpr int WB = TJ + 2, HB = TI + 2;   // stage B (zeta, alphaC)
    static constexpr int WC = TJ + 1, HC = TI + 1;   // R_C arrays and sigma12
    static constexpr int NZ = WZ * HZ, NB = WB * HB, NC = WC * HC;
    static constexpr int N_C_ARRAYS = 5 + (BASAL ? 1 : 0) + (SIDE ? 1 : 0);   // sig11 sig22 cd fvC fuC (cb) (sp)
    static constexpr size_t bytes() {
        return sizeof(T) * (size_t)(2 * NZ + (ADAPT ? 2 : 1) * NB + N_C_ARRAYS * NC);
    }
};

// rows [i0, i0 + ti) (ti <= TI) and columns [j0, j0 + 32) of one subcycle, by
// the NT threads of the CTA
template <class T, int TI, bool ADAPT, bool SIDE, bool BASAL, int NT = EVP_THREADS>
__device__ __forceinline__ void plain_tile(unsigned char *smem_raw, const Ctx<T> &c, const HaloFill &h,
                                           const EvpIO<T> &io, int i0, int ti, int j0) {
    using S = PlainSmem<T, TI, ADAPT, SIDE, BASAL>;
    T *e12s = reinterpret_cast<T *>(smem_raw);
    T *zqs = e12s + S::NZ;
    T *zeta = zqs + S::NZ;
    T *sig11 = zeta + S::NB;
    T *sig22 = sig11 + S::NC;
    T *cds = sig22 + S::NC;
    T *fvC = cds + S::NC;
    T *fuC = fvC + S::NC;
    T *cbs = fuC + S::NC;                      // basal drag only
    T *sps = cbs + (BASAL ? S::NC : 0);        // side drag only
    T *aCs = sps + (SIDE ? S::NC : 0);         // adaptive alpha only
    T *s12s = zqs;   // rAz*e12^2 is dead once stage B is done
    constexpr int TJ = S::TJ;
    const int nZ = (ti + 3) * S::WZ, nB = (ti + 2) * S::WB, nC = (ti + 1) * S::WC;

    const Fields<T> &f = c.f;
    const Dims &d = c.d;
    const int tid = threadIdx.x;

    // index helpers: stage A / B arrays are offset by one, R_C arrays by one,
    // R_Z (sigma12) by zero
#define ZA(li, lj) ((li) + 1) * S::WZ + ((lj) + 1)
#define ZB(li, lj) ((li) + 1) * S::WB + ((lj) + 1)
#define ZC(li, lj) ((li) + 1) * S::WC + ((lj) + 1)
#define ZZ(li, lj) (li) * S::WC + (lj)

    // ---- stage A: e12 at Z points
    for (int idx = tid; idx < nZ; idx += NT) {
        const int li = idx / S::WZ - 1, lj = idx % S::WZ - 1;
        const int gi = i0 + li, gj = j0 + lj;
        if (gi >= d.NX + 2 || gj >= d.NY + 2) continue;   // feeds no stored point; keeps the wrap within one period
        const T e = strain_z(c, io.u, io.v, gi, gj);
        e12s[idx] = e;
        zqs[idx] = c.ld(f.rAz, gi, gj) * (e * e);
    }
    __syncthreads();

    // ---- stage B: viscosities and the C-point stress update
    const T alpha = T(c.p.evpAlpha);
    const T rdenom = T(1.0 / c.p.evpAlpha);
    for (int idx = tid; idx < nB; idx += NT) {
        const int li = idx / S::WB - 1, lj = idx % S::WB - 1;
        const int gi = i0 + li, gj = j0 + lj;
        if (gi >= d.NX + 2 || gj >= d.NY + 2) continue;   // feeds no stored point; keeps the wrap within one period
        T e11, e22;
        strain_c(c, io.u, io.v, gi, gj, e11, e22);
        T zt, et, pr, dl;
        viscosity_c(c, gi, gj, e11, e22, zqs[ZA(li, lj)], zqs[ZA(li + 1, lj)], zqs[ZA(li, lj + 1)],
                    zqs[ZA(li + 1, lj + 1)], zt, et, pr, dl);
        zeta[idx] = zt;
        const T mC = c.ld(f.iceMask, gi, gj);
        T aC = alpha, d1 = rdenom;
        if (ADAPT) {
            const T mass = c.ld(f.SeaIceMassC, gi, gj);
            aC = sqrt(zt * T(c.p.EVPcFac) / (mass > T(1e-4) ? mass : T(1e-4)) * c.ld(f.recip_rA, gi, gj)) * mC;
            aC = aC > T(c.p.aEVPalphaMin) ? aC : T(c.p.aEVPalphaMin);
            aCs[idx] = aC;
            d1 = T(1.0) / aC;
        }
        if (li < ti && lj < TJ) {
            const int k = ZC(li, lj);
            const T ep = e11 + e22, em = e11 - e22;
            const T div = T(2) * zt * ep - pr;
            const T ten = T(2) * zt * em;
            const T s1 = (c.st(io.s1, gi, gj) * (aC - T(1)) + div) * d1 * mC;
            const T s2 = (c.st(io.s2, gi, gj) * (aC - T(1)) + ten * T(0.25)) * d1 * mC;
            sig11[k] = T(0.5) * (s1 + s2);
            sig22[k] = T(0.5) * (s1 - s2);
            if (li >= 0 && lj >= 0 && gi < d.NX && gj < d.NY) {
                const int64_t o = d.raw(gi, gj);
                io.s1o[o] = s1;
                io.s2o[o] = s2;
                if (ADAPT && io.aCo) io.aCo[o] = aC;
            }
            cds[k] = ocean_drag_c(c, io.u, io.v, gi, gj);
            if (BASAL) cbs[k] = basal_drag_c(c, io.u, io.v, gi, gj);
            const T mf = c.ld(f.SeaIceMassC, gi, gj) * c.ld(f.fCori, gi, gj) * T(0.5);
            fvC[k] = mf * (c.st(io.v, gi, gj) + c.st(io.v, gi, gj + 1));
            fuC[k] = mf * (c.st(io.u, gi, gj) + c.st(io.u, gi + 1, gj));
            if (SIDE) sps[k] = ice_speed_c(c, io.u, io.v, gi, gj);
        }
    }
    __syncthreads();

    // ---- stage C: sigma12 at Z points
    for (int idx = tid; idx < nC; idx += NT) {
        const int li = idx / S::WC, lj = idx % S::WC;
        const int gi = i0 + li, gj = j0 + lj;
        if (gi >= d.NX + 2 || gj >= d.NY + 2) continue;   // feeds no stored point; keeps the wrap within one period
        const T zz = c2z_norm(c, gi, gj, true) *
                     ((zeta[ZB(li, lj)] + zeta[ZB(li - 1, lj)]) + (zeta[ZB(li, lj - 1)] + zeta[ZB(li - 1, lj - 1)]));
        T aZ = alpha, d2 = rdenom;
        if (ADAPT) {
            aZ = T(0.5) * (T(0.5) * (aCs[ZB(li, lj)] + aCs[ZB(li, lj - 1)]) +
                           T(0.5) * (aCs[ZB(li - 1, lj)] + aCs[ZB(li - 1, lj - 1)]));
            d2 = T(1.0) / aZ;
        }
        const T shr = T(2) * zz * e12s[ZA(li, lj)];
        const T s12 = (c.st(io.s12, gi, gj) * (aZ - T(1)) + shr * T(0.25)) * d2;
        s12s[idx] = s12;
        if (li < ti && lj < TJ && gi < d.NX && gj < d.NY) io.s12o[d.raw(gi, gj)] = s12;
    }
    __syncthreads();

    chain_release();   // the next subcycle's CTAs may start; they wait for this launch's end

    // ---- stage D: momentum update at U and V points of the tile
    const T rdt = T(c.p.recip_deltatDyn);
    const T cosW = T(c.p.cosWat), sinW = T(c.p.sinWat);
    const T beta = T(c.p.evpBeta);
    for (int idx = tid; idx < ti * TJ; idx += NT) {
        const int li = idx / TJ, lj = idx % TJ;
        const int gi = i0 + li, gj = j0 + lj;
        if (gi >= d.NX || gj >= d.NY) continue;
        const int64_t o = d.raw(gi, gj);
        const T sg = sgn(__ldg(f.fCori + o));
        const T cd0 = cds[ZC(li, lj)], cdw = cds[ZC(li - 1, lj)], cdsou = cds[ZC(li, lj - 1)];
        const T cb0 = BASAL ? cbs[ZC(li, lj)] : T(0);
        const T cbw = BASAL ? cbs[ZC(li - 1, lj)] : T(0);
        const T cbs_ = BASAL ? cbs[ZC(li, lj - 1)] : T(0);
        const T u0 = io.u[o], v0 = io.v[o];

        // U point
        {
            const T sdx = (sig11[ZC(li, lj)] * __ldg(f.dyV + o) - sig11[ZC(li - 1, lj)] * c.ld(f.dyV, gi - 1, gj) -
                           s12s[ZZ(li, lj)] * __ldg(f.dxV + o) + s12s[ZZ(li, lj + 1)] * c.ld(f.dxV, gi, gj + 1)) *
                          __ldg(f.recip_rAu + o);
            const T mU = __ldg(f.SeaIceMassU + o);
            const T lm = mU != T(0) ? T(1) : mU;
            const T uo = __ldg(f.uOcean + o);
            const T du0 = uo - u0;
            const T dun = c.ld(f.uOcean, gi, gj + 1) - c.st(io.u, gi, gj + 1);
            const T duw = c.ld(f.uOcean, gi - 1, gj) - c.st(io.u, gi - 1, gj);
            const T duwn = c.ld(f.uOcean, gi - 1, gj + 1) - c.st(io.u, gi - 1, gj + 1);
            const T AW = __ldg(f.AreaW + o);
            T fx = __ldg(f.WindForcingX + o) +
                   (T(0.5) * (cd0 + cdw) * cosW * uo -
                    sg * sinW * T(0.5) * (cd0 * T(0.5) * (du0 + dun) + cdw * T(0.5) * (duw + duwn)) * lm) * AW;
            fx = fx + T(0.5) * (fvC[ZC(li, lj)] + fvC[ZC(li - 1, lj)]);
            const T bU = (ADAPT ? T(0.5) * (aCs[ZB(li, lj)] + aCs[ZB(li - 1, lj)]) : beta) * rdt;
            const T bU1 = bU + rdt;
            T den = mU * bU1 + AW * (T(0.5) * (cd0 + cdw) * cosW + T(0.5) * (cb0 + cbw));
            den = den == T(0) ? T(1) : den;
            if (SIDE) den = den + side_drag_u(c, gi, gj, sps[ZC(li, lj)], sps[ZC(li - 1, lj)]);
            const T un = __ldg(f.iceMaskU + o) * (bU * mU * u0 + mU * rdt * __ldg(io.uNm1 + o) + fx + sdx) / den;
            store_filled(io.uo, d, h, gi, gj, un);
        }
        // V point
        {
            const T sdy = (sig22[ZC(li, lj)] * __ldg(f.dxU + o) - sig22[ZC(li, lj - 1)] * c.ld(f.dxU, gi, gj - 1) -
                           s12s[ZZ(li, lj)] * __ldg(f.dyU + o) + s12s[ZZ(li + 1, lj)] * c.ld(f.dyU, gi + 1, gj)) *
                          __ldg(f.recip_rAv + o);
            const T mV = __ldg(f.SeaIceMassV + o);
            const T lm = mV != T(0) ? T(1) : mV;
            const T vo = __ldg(f.vOcean + o);
            const T dv0 = vo - v0;
            const T dve = c.ld(f.vOcean, gi + 1, gj) - c.st(io.v, gi + 1, gj);
            const T dvs = c.ld(f.vOcean, gi, gj - 1) - c.st(io.v, gi, gj - 1);
            const T dvse = c.ld(f.vOcean, gi + 1, gj - 1) - c.st(io.v, gi + 1, gj - 1);
            const T AS = __ldg(f.AreaS + o);
            T fy = __ldg(f.WindForcingY + o) +
                   (T(0.5) * (cd0 + cdsou) * cosW * vo +
                    sg * sinW * T(0.5) * (cd0 * T(0.5) * (dv0 + dve) + cdsou * T(0.5) * (dvs + dvse)) * lm) * AS;
            fy = fy - T(0.5) * (fuC[ZC(li, lj)] + fuC[ZC(li, lj - 1)]);
            const T bV = (ADAPT ? T(0.5) * (aCs[ZB(li, lj)] + aCs[ZB(li, lj - 1)]) : beta) * rdt;
            const T bV1 = bV + rdt;
            T den = mV * bV1 + AS * (T(0.5) * (cd0 + cdsou) * cosW + T(0.5) * (cb0 + cbs_));
            den = den == T(0) ? T(1) : den;
            if (SIDE) den = den + side_drag_v(c, gi, gj, sps[ZC(li, lj)], sps[ZC(li, lj - 1)]);
            const T vn = __ldg(f.iceMaskV + o) * (bV * mV * v0 + mV * rdt * __ldg(io.vNm1 + o) + fy + sdy) / den;
            store_filled(io.vo, d, h, gi, gj, vn);
        }
    }
#undef ZA
#undef ZB
#undef ZC
#undef ZZ
}

}  // namespace veris
