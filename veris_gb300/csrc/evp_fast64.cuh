// Float64 fast-form mEVP subcycle (veris/evp_solver.py:21-254), arranged for
// GB300's float64 pipe.
//
// GB300 executes float64 arithmetic at 2 lanes per SM and cycle, 1/64 of its
// float32 rate, so a float64 subcycle is bound by the number of float64-pipe
// instructions per cell (the HBM traffic is ~0.06 of the roofline).  The
// kernel computes the subcycle of the shared-memory tile in evp_tile.cuh
// (same stages, same wrap and halo semantics) with about half the float64
// instructions:
//
// * the 0/1 masks are applied as selects on the integer pipe, not as
//   multiplications; the wet-point count of the sigma12 average selects a
//   precomputed coefficient;
// * products of step constants are folded once per step by the prep
//   (recip_rA/e^2, mass*(beta+1)/dt, mass*beta/dt, 0.5*cos*Area, 0.25*m*f,
//   halved grid lengths, and 1/(2 alpha) into the ice strength factor, so
//   that its division by Delta + Delta_min gives zeta/(2 alpha), the stress
//   update's coefficient), one multiplication fewer per use; the drag
//   coefficient is the square root of the product the drag floor's test
//   forms;
// * divisions and square roots run in integer and float32 instructions
//   (f64math.cuh), of which the schedulers could issue ten times as many as
//   they do beside the float64 pipe: with the hardware's seeds and float64
//   series (four and five float64 operations each, 22 of 90 per cell)
//   1440 x 720 took 191 us a subcycle and 360 x 180 20.1, now 166 and 17.0; a
//   warp whose operands leave a safe exponent range uses IEEE division or
//   square root instead;
// * warps whose cells all have zero ice strength skip the viscosity's
//   square root and division (zeta = 0, which the formula gives), warps on
//   land skip the velocity division;
// * work units of at most 24 rows x 32 columns by default, three 256-thread
//   CTAs per SM (16 and 32 rows: four and two; the larger the unit, the
//   less ring work but the fewer resident warps to cover the float64 pipe's
//   latency), the launch ending on a round of small units so that the SMs
//   run out of work together.
//
// ADAPT: adaptive EVP (veris/evp_solver.py:65-73, 97-100, 148-150): alphaC
// from zeta at each C point in place of the constant alpha, its averages at
// Z, U and V.  SLIP: free slip with the side drag (veris/dynamics_routines.py:
// 99-140) in place of the no-slip boundary terms.  AUTO: the drop-in's loop;
// the prep has left in *a.viol whether the state is one that this form
// covers, and where it is not the CTA runs the plain tile instead.
#pragma once

#include "evp_fast.cuh"
#include "evp_plain.cuh"
#include "f64math.cuh"
#include "tile_units.cuh"

namespace veris {

struct F64Scalars {
    double am1r;             // (alpha - 1) / alpha
    double kp2;              // 2 * (press factor 2(1 - tsf)/(1 + tsf))
    double rsq, deltaMin;    // 1/e^2, Delta_min
    double dcq2N, dcq2S;     // 0.25 * (rhoSea * waterIceDrag)^2, north and south
    double cmin, cmin2;      // cDragMin, its square
    double U02;              // basal drag U0^2
    double sinW;             // sin(water turning angle)
    double nh1, nh2, nh3, nh4;   // 1 / n: the sigma12 average over n wet C points (of zeta / (2 alpha))
    double twoAlpha;             // 2 alpha: zeta from zeta / (2 alpha), for the tape
    double rdt, aMin, sideU0;    // 1/dt, aEVPalphaMin (adaptive EVP), sideDragU0 (free slip)
};

// the drop-in's loop: the state check's result and what the plain tile reads
struct F64Auto {
    const int *viol = nullptr;
    const Ctx<double> *ctx = nullptr;
    const double *sdU = nullptr, *sdV = nullptr;   // side drag: mass * sideDragCoeff * coastline factor (SLIP)
};

inline F64Scalars f64_scalars(const FastScalars<double> &k, double sideU0 = 0.0) {
    F64Scalars s;
    s.am1r = k.alpha_m1 * k.ralpha;
    s.kp2 = 2.0 * k.kp;
    s.rsq = k.rsq;
    s.deltaMin = k.deltaMin;
    s.dcq2N = 0.25 * k.dN2;
    s.dcq2S = 0.25 * k.dS2;
    s.cmin = k.cmin;
    s.cmin2 = k.cmin2;
    s.U02 = k.U02;
    s.sinW = k.sinW;
    s.nh1 = 1.0;
    s.nh2 = 0.5;
    s.nh3 = 1.0 / 3.0;
    s.nh4 = 0.25;
    s.twoAlpha = 2.0 / k.ralpha;
    s.rdt = k.rdt;
    s.aMin = k.aMin;
    s.sideU0 = sideU0;
    return s;
}

// ------------------------------------------------------------------ tile
constexpr int F64_THREADS = 256, F64_WIDE = 768;
constexpr int F64_LOOP_ROWS = 16;

// a loop of n subcycles: the first reads `in`, subcycle it < n - 1 writes
// `even` or `odd` (pitch of the inputs), the last `out` (pitch ldo)
struct F64Loop {
    const double *in[5];
    double *even[5], *odd[5], *out[5];
    int64_t ldo;
    int n;
    unsigned *arrived;   // zero at the launch
};

// Pieces of up to 8 rows in a CTA of 768 threads give its 24 warps fewer tasks
// than they could take (a 2-row piece has 5 for its viscosities, 2 for its
// velocities), and a scheduler's float64 pipe serves one warp instruction in 64
// cycles: two warps of 45 such instructions on one scheduler are the whole
// stage.  There the drag and Coriolis terms, and U and V points, are tasks of
// their own.  Per subcycle 90 x 40 8.5 -> 6.6 us, 180 x 90 9.0 -> 7.7,
// 240 x 121 10.7 -> 9.8; of 9 to 11 rows the warps are busy without and the
// index work is paid twice: 300 x 150 13.0 -> 13.9, 360 x 180 15.7 -> 16.7.
constexpr int F64_SPLIT_ROWS = 8;

// TI output rows x 32 columns per CTA; 16-, 24- and 32-row tiles fit 4, 3
// and 2 CTAs per SM (smaller tiles: more resident warps, more ring work)
template <int TI_>
struct Smem64 {
    static constexpr int TI = TI_, TJ = 32;
    static constexpr int WS = TJ + 4, HS = TI + 4, NS = WS * HS;   // u, v, flags: origin -2
    static constexpr int WZ = TJ + 3, HZ = TI + 3, NZ = WZ * HZ;   // e12 and rAz*e12^2: origin -1
    static constexpr int WB = TJ + 2, HB = TI + 2, NB = WB * HB;   // zeta: origin -1
    static constexpr int WC = TJ + 1, HC = TI + 1, NC = WC * HC;   // C ring (origin -1), Z (origin 0)
    static constexpr size_t bytes(bool basal, bool adapt = false, bool slip = false) {
        return sizeof(double) * (size_t)(2 * NS + 2 * NZ + (adapt ? 2 : 1) * NB +
                                         (5 + (basal ? 1 : 0) + (slip ? 1 : 0)) * NC) +
               sizeof(uint32_t) * NS;
    }
};
constexpr int f64_min_blocks(int ti) { return ti <= 16 ? 4 : (ti <= 24 ? 3 : 2); }
static_assert(2 * (Smem64<32>::bytes(true) + 1024) <= 228 * 1024, "two 32-row CTAs per SM");
static_assert(3 * (Smem64<24>::bytes(false) + 1024) <= 228 * 1024, "three 24-row CTAs per SM");
static_assert(4 * (Smem64<16>::bytes(true) + 1024) <= 228 * 1024, "four 16-row CTAs per SM");
static_assert(3 * (Smem64<16>::bytes(true, true, true) + 1024) <= 228 * 1024, "three 16-row CTAs with every option");

// The plain tile in a CTA of the folded form's launch: the settings and field
// table come through shared memory behind the tile's arrays.  Not inlined:
// the folded form keeps its registers.
template <int TI, bool ADAPT, bool SLIP, bool BASAL, int NT>
__device__ __noinline__ void plain_fallback(const Ctx<double> *ctx, HaloFill h, FastIO<double> io, int i0, int ti,
                                            int j0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr size_t at = (PlainSmem<double, TI, ADAPT, SLIP, BASAL>::bytes() + 15) / 16 * 16;
    static_assert(at + sizeof(Ctx<double>) <= Smem64<TI>::bytes(BASAL, ADAPT, SLIP), "the plain tile's shared memory");
    Ctx<double> *c = reinterpret_cast<Ctx<double> *>(smem_raw + at);
    static_assert(sizeof(Ctx<double>) % sizeof(int) == 0, "copied by words");
    for (int q = threadIdx.x; q < (int)(sizeof(Ctx<double>) / sizeof(int)); q += NT)
        reinterpret_cast<int *>(c)[q] = reinterpret_cast<const int *>(ctx)[q];
    __syncthreads();
    const EvpIO<double> p{io.u, io.v, io.s1, io.s2, io.s12, io.uo, io.vo, io.s1o, io.s2o, io.s12o,
                          c->f.uIce, c->f.vIce, io.aCo};
    plain_tile<double, TI, ADAPT, SLIP, BASAL, NT>(smem_raw, *c, h, p, i0, ti, j0);
}

// rows [i0, i0 + ti) and the 32 columns from j0 of one subcycle.  LOOP: one of
// a launch that runs the whole loop (no successor to start)
template <int TI, bool BASAL, bool TURN, bool TAPE, bool ADAPT, bool SLIP, bool AUTO, int NT, bool LOOP>
__device__ __forceinline__ void f64_tile(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c,
                                         const F64Scalars &k, const FastIO<double> &io, const F64Auto &a, int i0,
                                         int ti, int j0) {
    using S = Smem64<TI>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sU = reinterpret_cast<double *>(smem_raw);
    double *sV = sU + S::NS;
    double *sE12 = sV + S::NS;
    double *sZq = sE12 + S::NZ;   // rAz*e12^2 in stages A/B, then sigma12 (origin 0, pitch WC)
    double *sZeta = sZq + S::NZ;
    double *sS11 = sZeta + S::NB;
    double *sS22 = sS11 + S::NC;
    double *sCd = sS22 + S::NC;
    double *sFv = sCd + S::NC;
    double *sFu = sFv + S::NC;
    double *sCb = sFu + S::NC;    // basal drag only
    double *sSp = sCb + (BASAL ? S::NC : 0);   // ice speed, side drag only
    double *sA = sSp + (SLIP ? S::NC : 0);     // adaptive alpha only
    uint32_t *sF = reinterpret_cast<uint32_t *>(sA + (ADAPT ? S::NB : 0));
    double *sS12 = sZq;
    // the unit's region sizes (ti <= TI rows)
    const int nS = (ti + 4) * S::WS, nZ = (ti + 3) * S::WZ, nB = (ti + 2) * S::WB, nC = (ti + 1) * S::WC;
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr unsigned ALL = 0xffffffffu;
#define IS(li, lj) (((li) + 2) * S::WS + ((lj) + 2))
#define IZ(li, lj) (((li) + 1) * S::WZ + ((lj) + 1))
#define IB(li, lj) (((li) + 1) * S::WB + ((lj) + 1))
#define IC(li, lj) (((li) + 1) * S::WC + ((lj) + 1))
#define IZZ(li, lj) ((li) * S::WC + (lj))
    const bool split = NT == F64_WIDE && ti <= F64_SPLIT_ROWS;
    // ocean velocities at tile offsets (read through L1; not staged)
    auto uoc = [&](int li, int lj) { return __ldg(c.uOc + (int64_t)d.wxt(i0 + li) * lp + d.wyt(j0 + lj)); };
    auto voc = [&](int li, int lj) { return __ldg(c.vOc + (int64_t)d.wxt(i0 + li) * lp + d.wyt(j0 + lj)); };

    // ---- stage u, v and the flags of the tile plus a 2-cell ring
    for (int idx = tid; idx < nS; idx += NT) {
        const int li = idx / S::WS - 2, lj = idx % S::WS - 2;
        const int64_t o = (int64_t)d.wxt(i0 + li) * lp + d.wyt(j0 + lj);
        sU[idx] = io.u[o];
        sV[idx] = io.v[o];
        sF[idx] = __ldg(c.flags + o);
    }
    __syncthreads();

    // ---- A: e12 at Z points [-1, TI+1] x [-1, TJ+1] (veris/dynamics_routines.py:160-175)
    for (int base = 0; base < nZ; base += NT) {
        const int idx = base + tid;
        const unsigned m = __ballot_sync(ALL, idx < nZ);
        if (idx >= nZ) continue;
        const int li = idx / S::WZ - 1, lj = idx % S::WZ - 1;
        const int gi = d.wxt(i0 + li), gj = d.wyt(j0 + lj);
        const uint32_t f0 = sF[IS(li, lj)], fw = sF[IS(li - 1, lj)], fs = sF[IS(li, lj - 1)],
                       fws = sF[IS(li - 1, lj - 1)];
        const bool mz = (f0 & fw & fs & fws & F_MC) != 0;
        // no-slip boundary terms: (iceMaskU - its southern neighbour) and (iceMaskV - its western one)
        const int hU = (int)((f0 & F_MU) != 0) - (int)((fs & F_MU) != 0);
        const int hV = (int)((f0 & F_MV) != 0) - (int)((fw & F_MV) != 0);
        const double u0 = sU[IS(li, lj)], us = sU[IS(li, lj - 1)];
        const double v0 = sV[IS(li, lj)], vw = sV[IS(li - 1, lj)];
        const double ry = __ldg(c.rdyUh_y + gj), rx = __ldg(c.rdxVh_x + gi);
        double e;
        if (!SLIP && __any_sync(m, (hU | hV) != 0)) {
            const double hu2 = hU == 0 ? 0.0 : (hU > 0 ? 2.0 : -2.0);
            const double hv2 = hV == 0 ? 0.0 : (hV > 0 ? 2.0 : -2.0);
            const double tu = fma(hu2, u0 + us, mz ? u0 - us : 0.0);
            const double tv = fma(hv2, v0 + vw, mz ? v0 - vw : 0.0);
            e = fma(ry, tu, rx * tv);
        } else {
            e = mz ? fma(ry, u0 - us, rx * (v0 - vw)) : 0.0;
        }
        sE12[idx] = e;
        sZq[idx] = __ldg(c.rAz + (int64_t)gi * lp + gj) * (e * e);
    }
    __syncthreads();

    // ---- B: viscosities at C [-1, TI] x [-1, TJ] (veris/dynamics_routines.py:220-268);
    //      stresses, drag and Coriolis terms on [-1, TI) x [-1, TJ) (veris/evp_solver.py:80-145)
    auto drag_terms = [&](unsigned m2, int li, int lj, int gi, int gj, int64_t o, uint32_t f0, double u0, double ue,
                          double v0, double vn, bool own) {
        const int q = IC(li, lj);
        const bool mC = f0 & F_MC;
        // ocean drag at C (veris/dynamics_routines.py:21-52): with X = 4 t and
        // Y = (dc^2/4) X, dc^2 t > cmin^2 <=> Y > cmin^2 and dc sqrt(t) = sqrt(Y)
        const uint32_t fe = sF[IS(li + 1, lj)], fn = sF[IS(li, lj + 1)];
        const double du0 = (f0 & F_INU) ? u0 - __ldg(c.uOc + o) : 0.0;
        const double du1 = (fe & F_INU) ? ue - uoc(li + 1, lj) : 0.0;
        const double dv0 = (f0 & F_INV) ? v0 - __ldg(c.vOc + o) : 0.0;
        const double dv1 = (fn & F_INV) ? vn - voc(li, lj + 1) : 0.0;
        const double a = du0 + du1, b = dv0 + dv1;
        const double X = fma(b, b, a * a);
        const bool south = f0 & F_SOUTH;
        const double Y = (south ? k.dcq2S : k.dcq2N) * X;
        const bool fast = gt_nonneg(Y, k.cmin2);
        double cd = k.cmin;
        if (__any_sync(m2, fast)) {
            const double sy = sqrt64(Y, m2);
            if (fast) cd = sy;
        }
        sCd[q] = mC ? cd : 0.0;
        if (TAPE && own) io.tCd[(int64_t)gi * io.ldo + gj] = mC ? cd : 0.0;
        if (BASAL) {   // veris/dynamics_routines.py:55-96 with the step factor folded by the prep
            const double a_ = (f0 & F_INU) ? u0 : 0.0, b_ = (fe & F_INU) ? ue : 0.0;
            const double c_ = (f0 & F_INV) ? v0 : 0.0, e_ = (fn & F_INV) ? vn : 0.0;
            const double s = 0.25 * (a_ * a_ + b_ * b_ + c_ * c_ + e_ * e_);
            sCb[q] = div64(__ldg(c.bfac + o), sqrt64(s + k.U02, m2), m2);
        }
        const double mf = __ldg(c.mf4 + o);
        sFv[q] = mf * (v0 + vn);
        sFu[q] = mf * (u0 + ue);
        if (SLIP) {   // veris/dynamics_routines.py:110-112
            const double us = u0 + ue, vs = v0 + vn;
            sSp[q] = 0.5 * sqrt64(fma(us, us, vs * vs), m2);
        }
    };
    const int firstD = (nB + 31) / 32 * 32;   // the first drag task's threads
    for (int base = 0; base < (split ? firstD + nC : nB); base += NT) {
        const int idx = base + tid;
        if (NT == F64_WIDE && split && idx >= firstD) {   // the drag and Coriolis terms of 32 points
            const int q = idx - firstD;
            const unsigned m2 = __ballot_sync(ALL, q < nC);
            if (q >= nC) continue;
            const int li = q / S::WC - 1, lj = q % S::WC - 1;
            const int gi = d.wxt(i0 + li), gj = d.wyt(j0 + lj);
            drag_terms(m2, li, lj, gi, gj, (int64_t)gi * lp + gj, sF[IS(li, lj)], sU[IS(li, lj)],
                       sU[IS(li + 1, lj)], sV[IS(li, lj)], sV[IS(li, lj + 1)],
                       li >= 0 && lj >= 0 && i0 + li < d.NX && j0 + lj < d.NY);
            continue;
        }
        const unsigned m = __ballot_sync(ALL, idx < nB);
        if (idx >= nB) continue;
        const int li = idx / S::WB - 1, lj = idx % S::WB - 1;
        const int gi = d.wxt(i0 + li), gj = d.wyt(j0 + lj);
        const int64_t o = (int64_t)gi * lp + gj;
        const uint32_t f0 = sF[IS(li, lj)];
        const bool inC = f0 & F_INC;
        const double u0 = sU[IS(li, lj)], ue = sU[IS(li + 1, lj)];
        const double v0 = sV[IS(li, lj)], vn = sV[IS(li, lj + 1)];
        const double e11 = inC ? (ue - u0) * __ldg(c.rdxU_x + gi) : 0.0;
        const double e22 = inC ? (vn - v0) * __ldg(c.rdyV_y + gj) : 0.0;
        const double ep = e11 + e22, em = e11 - e22;
        // constant alpha: Ph / (2 alpha), and zeta below is zeta / (2 alpha)
        const double Ph = __ldg((ADAPT ? c.Ph : c.Phh) + o);
        double zeta = 0.0, delta = 0.0;
        // (a taped subcycle keeps Delta where zeta = 0 too: the adjoint needs it)
        const bool strong = __any_sync(m, !is_zero(Ph));
        if (TAPE || strong) {
            const double zs =
                (sZq[IZ(li, lj)] + sZq[IZ(li + 1, lj)]) + (sZq[IZ(li, lj + 1)] + sZq[IZ(li + 1, lj + 1)]);
            // Delta^2 = ep^2 + (em^2 + 4 * 0.25/rA * sum rAz e12^2) / e^2
            const double d2 = fma(__ldg(c.rsqrA + o), zs, fma(k.rsq * em, em, ep * ep));
            delta = sqrt64(d2, m);
            if (strong) zeta = div64(Ph, delta + k.deltaMin, m);
        }
        sZeta[idx] = zeta;
        double aC = 0.0;
        if (ADAPT) {
            const double x = zeta * __ldg(c.acf + o);
            const double r = strong ? sqrt64(x, m) : 0.0;   // every lane of m
            aC = (f0 & F_MC) ? r : 0.0;
            aC = aC > k.aMin ? aC : k.aMin;
            sA[idx] = aC;
        }
        const bool in2 = li < ti && lj < S::TJ;
        const unsigned m2 = __ballot_sync(m, in2);
        if (in2) {
            const int q = IC(li, lj);
            const bool mC = f0 & F_MC;
            // sigma_k = sigma_k (alpha-1)/alpha + zeta/(2 alpha) * (4 ep - 2 kp Delta | em)
            const double ra = ADAPT ? div64(1.0, aC, m2) : 0.0;
            const double zh = ADAPT ? 0.5 * zeta * ra : zeta;
            const double am1r = ADAPT ? (aC - 1.0) * ra : k.am1r;
            const double s1 = mC ? fma(io.s1[o], am1r, zh * fma(4.0, ep, -(k.kp2 * delta))) : 0.0;
            const double s2 = mC ? fma(io.s2[o], am1r, zh * em) : 0.0;
            sS11[q] = (s1 + s2) * __ldg(c.dyVh_y + gj);
            sS22[q] = (s1 - s2) * __ldg(c.dxUh_x + gi);
            const bool own = li >= 0 && lj >= 0 && i0 + li < d.NX && j0 + lj < d.NY;
            if (own) {
                const int64_t w = (int64_t)gi * io.ldo + gj;
                io.s1o[w] = s1;
                io.s2o[w] = s2;
                if (AUTO && ADAPT && io.aCo) io.aCo[w] = aC;
                if (TAPE) {
                    io.tDel[w] = delta;
                    io.tZeta[w] = zeta * k.twoAlpha;
                }
            }
            if (!split) drag_terms(m2, li, lj, gi, gj, o, f0, u0, ue, v0, vn, own);
        }
    }
    __syncthreads();

    // ---- C: sigma12 at Z [0, TI] x [0, TJ] (veris/evp_solver.py:101-103 with
    //      veris/averaging.py:4-19); sZq is dead: it takes sigma12
    for (int idx = tid; idx < nC; idx += NT) {
        const int li = idx / S::WC, lj = idx % S::WC;
        const int gi = d.wxt(i0 + li), gj = d.wyt(j0 + lj);
        const uint32_t n = (sF[IS(li, lj)] & F_MC) + (sF[IS(li - 1, lj)] & F_MC) + (sF[IS(li, lj - 1)] & F_MC) +
                           (sF[IS(li - 1, lj - 1)] & F_MC);
        const double nh = n == 4 ? k.nh4 : (n == 3 ? k.nh3 : (n == 2 ? k.nh2 : (n == 1 ? k.nh1 : 0.0)));
        const double zs = (sZeta[IB(li, lj)] + sZeta[IB(li - 1, lj)]) +
                          (sZeta[IB(li, lj - 1)] + sZeta[IB(li - 1, lj - 1)]);
        double s12 = io.s12[(int64_t)gi * lp + gj];
        if (ADAPT) {
            const double aZ = 0.25 * ((sA[IB(li, lj)] + sA[IB(li, lj - 1)]) + (sA[IB(li - 1, lj)] + sA[IB(li - 1, lj - 1)]));
            s12 = fma(s12, aZ - 1.0, (0.5 * nh * zs) * sE12[IZ(li, lj)]) * rcp_lane(aZ);
        } else {
            s12 = fma(s12, k.am1r, (nh * zs) * sE12[IZ(li, lj)]);
        }
        sS12[idx] = s12;
        if (li < ti && lj < S::TJ && i0 + li < d.NX && j0 + lj < d.NY) io.s12o[(int64_t)gi * io.ldo + gj] = s12;
    }
    __syncthreads();

    // the next subcycle's CTAs may start: they find room as this launch's last
    // CTAs end, and stage D covers their launch latency (released before D
    // 191.0 us a subcycle on 1440 x 720, before C 191.4, before B 191.1, at
    // the kernel's start 192.1, unchained 194.0; 360 x 180: 20.1, 20.5, 20.8,
    // 21.2, 22.6)
    if (!LOOP) chain_release();

    // ---- D: u, v at the tile's U and V points (veris/evp_solver.py:105-187)
    for (int t = tid >> 5; t < (split ? 2 * ti : ti); t += NT / 32) {   // a row's U and V points, or one of the two
        const bool doU = t < ti, doV = !split || !doU;
        const int li = doU ? t : t - ti, lj = lane;
        const int gi = i0 + li, gj = j0 + lj;
        const bool act = gi < d.NX && gj < d.NY;
        const unsigned m = __ballot_sync(ALL, act);
        if (!act) continue;
        const int64_t o = (int64_t)gi * lp + gj;
        const uint32_t f0 = sF[IS(li, lj)];
        const double u0 = sU[IS(li, lj)], v0 = sV[IS(li, lj)];
        const double cd0 = sCd[IC(li, lj)], cdw = sCd[IC(li - 1, lj)], cds = sCd[IC(li, lj - 1)];
        if (doU) {   // U point
            const double kU = __ldg(c.hAW + o) * (cd0 + cdw);
            const double uo0 = __ldg(c.uOc + o);
            double fx = fma(kU, uo0, __ldg(c.cU + o)) + (sFv[IC(li, lj)] + sFv[IC(li - 1, lj)]);
            if (TURN) {
                const double sg = (f0 & F_SPOS) ? 1.0 : ((f0 & F_SNEG) ? -1.0 : 0.0);
                const double du0 = uo0 - u0, dun = uoc(li, lj + 1) - sU[IS(li, lj + 1)];
                const double duw = uoc(li - 1, lj) - sU[IS(li - 1, lj)];
                const double duwn = uoc(li - 1, lj + 1) - sU[IS(li - 1, lj + 1)];
                const double t = (cd0 * 0.5 * (du0 + dun) + cdw * 0.5 * (duw + duwn)) * __ldg(c.AW + o);
                if (f0 & F_LMU) fx -= sg * k.sinW * 0.5 * t;
            }
            const double sdx = __ldg(c.rrAu + o) * fma(__ldg(c.dxV_x + gi), sS12[IZZ(li, lj + 1)] - sS12[IZZ(li, lj)],
                                                       sS11[IC(li, lj)] - sS11[IC(li - 1, lj)]);
            double mUb, mUb1;
            if (ADAPT) {
                const double mU = __ldg(c.mU + o);
                mUb = mU * (0.5 * (sA[IB(li, lj)] + sA[IB(li - 1, lj)]) * k.rdt);
                mUb1 = fma(mU, k.rdt, mUb);
            } else {
                mUb = __ldg(c.mUb + o);
                mUb1 = __ldg(c.mUb1 + o);
            }
            double den = mUb1 + kU;
            if (BASAL) den = fma(0.5 * __ldg(c.AW + o), sCb[IC(li, lj)] + sCb[IC(li - 1, lj)], den);
            den = is_zero(den) ? 1.0 : den;
            if (SLIP) {
                const double sp = __ldg(c.AW + o) > 0.0 ? 0.5 * (sSp[IC(li, lj)] + sSp[IC(li - 1, lj)]) : 0.0;
                den += div64(__ldg(a.sdU + o), sp + k.sideU0, m);
            }
            const double num = fma(mUb, u0, fx) + sdx;
            const bool wet = f0 & F_MU;
            double un = 0.0;
            if (__any_sync(m, wet)) {
                const double q = div64(num, den, m);
                un = wet ? q : 0.0;
            }
            store_filled_ld(io.uo, io.ldo, d, h, gi, gj, un);
        }
        if (doV) {   // V point
            const double kV = __ldg(c.hAS + o) * (cd0 + cds);
            const double vo0 = __ldg(c.vOc + o);
            double fy = fma(kV, vo0, __ldg(c.cV + o)) - (sFu[IC(li, lj)] + sFu[IC(li, lj - 1)]);
            if (TURN) {
                const double sg = (f0 & F_SPOS) ? 1.0 : ((f0 & F_SNEG) ? -1.0 : 0.0);
                const double dv0 = vo0 - v0, dve = voc(li + 1, lj) - sV[IS(li + 1, lj)];
                const double dvs = voc(li, lj - 1) - sV[IS(li, lj - 1)];
                const double dvse = voc(li + 1, lj - 1) - sV[IS(li + 1, lj - 1)];
                const double t = (cd0 * 0.5 * (dv0 + dve) + cds * 0.5 * (dvs + dvse)) * __ldg(c.AS + o);
                if (f0 & F_LMV) fy += sg * k.sinW * 0.5 * t;
            }
            const double sdy = __ldg(c.rrAv + o) * fma(__ldg(c.dyU_y + gj), sS12[IZZ(li + 1, lj)] - sS12[IZZ(li, lj)],
                                                       sS22[IC(li, lj)] - sS22[IC(li, lj - 1)]);
            double mVb, mVb1;
            if (ADAPT) {
                const double mV = __ldg(c.mV + o);
                mVb = mV * (0.5 * (sA[IB(li, lj)] + sA[IB(li, lj - 1)]) * k.rdt);
                mVb1 = fma(mV, k.rdt, mVb);
            } else {
                mVb = __ldg(c.mVb + o);
                mVb1 = __ldg(c.mVb1 + o);
            }
            double den = mVb1 + kV;
            if (BASAL) den = fma(0.5 * __ldg(c.AS + o), sCb[IC(li, lj)] + sCb[IC(li, lj - 1)], den);
            den = is_zero(den) ? 1.0 : den;
            if (SLIP) {
                const double sp = __ldg(c.AS + o) > 0.0 ? 0.5 * (sSp[IC(li, lj)] + sSp[IC(li, lj - 1)]) : 0.0;
                den += div64(__ldg(a.sdV + o), sp + k.sideU0, m);
            }
            const double num = fma(mVb, v0, fy) + sdy;
            const bool wet = f0 & F_MV;
            double vnew = 0.0;
            if (__any_sync(m, wet)) {
                const double q = div64(num, den, m);
                vnew = wet ? q : 0.0;
            }
            store_filled_ld(io.vo, io.ldo, d, h, gi, gj, vnew);
        }
    }
#undef IS
#undef IZ
#undef IB
#undef IC
#undef IZZ
}

template <int TI, bool BASAL, bool TURN, bool TAPE, bool ADAPT, bool SLIP, bool AUTO, int NT>
__global__ void __launch_bounds__(NT, NT > F64_THREADS ? 1 : ((ADAPT || SLIP) ? 3 : f64_min_blocks(TI)))
evp_f64_kernel(Dims d, int64_t lp, HaloFill h, FastConsts<double> c, F64Scalars k, FastIO<double> io,
               TileUnits w, F64Auto a) {
    int i0, ti, j0;
    w.unit(blockIdx.x, d.NX, i0, ti, j0);
    chain_wait();
    if (AUTO) {
        if (*a.viol) {   // the same for every CTA and subcycle
            plain_fallback<TI, ADAPT, SLIP, BASAL, NT>(a.ctx, h, io, i0, ti, j0);
            return;
        }
    }
    f64_tile<TI, BASAL, TURN, TAPE, ADAPT, SLIP, AUTO, NT, false>(d, lp, h, c, k, io, a, i0, ti, j0);
}

// the n subcycles of a unit, `tile` one of them; false if a barrier gave up
template <class F>
__device__ __forceinline__ bool f64_loop(const F64Loop &l, int64_t lp, F tile) {
    FastIO<double> io{l.in[0], l.in[1], l.in[2], l.in[3], l.in[4]};
    for (int it = 0;; ++it) {
        const bool last = it == l.n - 1;
        double *const *to = last ? l.out : (it & 1 ? l.odd : l.even);
        io.uo = to[0];
        io.vo = to[1];
        io.s1o = to[2];
        io.s2o = to[3];
        io.s12o = to[4];
        io.ldo = last ? l.ldo : lp;
        tile(io);
        if (last) return true;
        if (!grid_barrier(l.arrived, it + 1)) return false;
        io.u = io.uo;
        io.v = io.vo;
        io.s1 = io.s1o;
        io.s2 = io.s2o;
        io.s12 = io.s12o;
    }
}

// A whole loop of n subcycles in one launch, one unit per CTA.  The barrier
// between two subcycles takes what starting the next of a chain of launches
// takes or a little more (a subcycle on 90 x 40 6.7 us chained, 6.7 so,
// 180 x 90 7.8 and 8.0, 240 x 121 10.0 and 10.0, 360 x 180 15.5 and 15.7).
// What goes is the host's 5.5 us per launch, which a chain of short subcycles
// does not cover once the host has more to do: a step on 90 x 40 with 120 of
// them takes 1066 us instead of 1393.
template <bool BASAL, bool TURN, bool ADAPT, bool SLIP>
__global__ void __launch_bounds__(F64_WIDE, 1)
evp_f64_loop_kernel(Dims d, int64_t lp, HaloFill h, FastConsts<double> c, F64Scalars k, F64Loop l, TileUnits w,
                    F64Auto a) {
    constexpr int TI = F64_LOOP_ROWS, NT = F64_WIDE;
    int i0, ti, j0;
    w.unit(blockIdx.x, d.NX, i0, ti, j0);
    bool done;
    if (*a.viol)
        done = f64_loop(l, lp, [&](const FastIO<double> &io) {
            plain_fallback<TI, ADAPT, SLIP, BASAL, NT>(a.ctx, h, io, i0, ti, j0);
        });
    else
        done = f64_loop(l, lp, [&](const FastIO<double> &io) {
            f64_tile<TI, BASAL, TURN, false, ADAPT, SLIP, true, NT, true>(d, lp, h, c, k, io, a, i0, ti, j0);
        });
    if (done) return;
    for (int q = threadIdx.x; q < ti * 32; q += NT) {   // given up: no number stands for a result
        const int gi = i0 + q / 32, gj = j0 + q % 32;
        if (gi < d.NX && gj < d.NY)
            for (int f = 0; f < 5; ++f)
                l.out[f][(int64_t)gi * l.ldo + gj] = __longlong_as_double(0x7ff8000000000000ll);
    }
}

template <int TI, bool B, bool R, bool TP, bool AD, bool SL, bool AUTO, int NT>
static int launch64_tile(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c, const F64Scalars &k,
                    const FastIO<double> &io, cudaStream_t st, const F64Auto &a) {
    using S = Smem64<TI>;
    auto kern = evp_f64_kernel<TI, B, R, TP, AD, SL, AUTO, NT>;
    const size_t sm = S::bytes(B, AD, SL);
    static std::atomic<bool> configured[MAX_DEVICES];
    if (!smem_configured(configured, kern, (int)sm)) return VERIS_ERR_LAUNCH;
    static std::atomic<int> resident[MAX_DEVICES];
    const int slots = cta_slots(resident, kern, NT, sm);
    if (slots <= 0) return VERIS_ERR_LAUNCH;
    if (NT == F64_WIDE && (int64_t)((d.NY + S::TJ - 1) / S::TJ) * ((d.NX + TI - 1) / TI) > slots)
        return VERIS_ERR_UNSUPPORTED;
    const TileUnits w = tile_units(d, TI, slots);
    return launch_chained(kern, dim3(w.count), dim3(NT), sm, st, d, lp, h, c, k, io, w, a);
}

// Grids that one 16-row piece per SM covers take one CTA of 768 threads per SM:
// as many warps as three of 256, on pieces three times as tall, whose rings are
// a smaller part of the work.  Per subcycle, three CTAs / one (without split
// tasks): 128 x 64 10.4 / 8.6 us, 180 x 90 11.0 / 9.0, 240 x 121 12.3 / 10.7,
// 360 x 180 17.1 / 15.8; with taller pieces the three win, 443 x 221 23.5 / 25.0,
// 600 x 300 35.0 / 45.6.
// (384 threads x 2: 9.5, 9.5, 11.5, 16.9; 512 x 1: 8.4, 8.7, 10.5, 18.9.)
template <int TI, bool B, bool R, bool TP, bool AD = false, bool SL = false, bool AUTO = false>
static int launch64(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c, const F64Scalars &k,
                    const FastIO<double> &io, cudaStream_t st, const F64Auto &a = F64Auto{}) {
    const int stt = launch64_tile<F64_LOOP_ROWS, B, R, TP, AD, SL, AUTO, F64_WIDE>(d, lp, h, c, k, io, st, a);
    if (stt != VERIS_ERR_UNSUPPORTED) return stt;
    return launch64_tile<TI, B, R, TP, AD, SL, AUTO, F64_THREADS>(d, lp, h, c, k, io, st, a);
}

// The drop-in's loop in one launch, where the pieces are short enough that the
// host's time per launch shows (evp_f64_loop_kernel); VERIS_ERR_UNSUPPORTED,
// having launched nothing, on larger grids.
template <bool B, bool R, bool AD, bool SL>
static int launch64_loop(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c,
                         const F64Scalars &k, const F64Loop &l, cudaStream_t st, const F64Auto &a) {
    using S = Smem64<F64_LOOP_ROWS>;
    auto kern = evp_f64_loop_kernel<B, R, AD, SL>;
    const size_t sm = S::bytes(B, AD, SL);
    static std::atomic<bool> configured[MAX_DEVICES];
    if (!smem_configured(configured, kern, (int)sm)) return VERIS_ERR_LAUNCH;
    static std::atomic<int> resident[MAX_DEVICES];
    const int slots = cta_slots(resident, kern, F64_WIDE, sm);
    if (slots <= 0) return VERIS_ERR_LAUNCH;
    if ((int64_t)((d.NY + S::TJ - 1) / S::TJ) * ((d.NX + F64_LOOP_ROWS - 1) / F64_LOOP_ROWS) > slots)
        return VERIS_ERR_UNSUPPORTED;
    const TileUnits w = tile_units(d, F64_LOOP_ROWS, slots);
    if ((d.NX + w.P1 - 1) / w.P1 > F64_SPLIT_ROWS) return VERIS_ERR_UNSUPPORTED;
    return launch_cooperative(kern, dim3(w.count), dim3(F64_WIDE), sm, st, d, lp, h, c, k, l, w, a);
}

}  // namespace veris
