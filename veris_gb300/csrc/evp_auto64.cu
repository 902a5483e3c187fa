// The drop-in's float64 subcycle loop (veris/evp_solver.py:257-319): the folded
// form of evp_fast64.cuh on the caller's own arrays, any state.
//
// The plain loop (evp.cu) evaluates every option with the reference's order of
// operations and IEEE division: 210 float64 operations per cell and subcycle
// and more against the folded form's 90, on a GPU whose float64 pipe is what
// binds.  Per subcycle, plain (32-row tiles) / folded:
//   90 x 40      104 / 6.7 us    with adaptive, side, basal and turned terms 183 / 9.0
//   360 x 180    104 / 15.6                                                  185 / 26.6
//   1440 x 720   690 / 167                                                 1092 / 320
// and 19, 60, 657 us (30, 96, 1022) on states left to the plain tile.  Whether a state is one the
// folded form covers (metrics that vary along one axis, masks 0 or 1, no
// curvature terms, finite inputs) is only known on the device, so the once-per-
// call preparation, which reads every field anyway, leaves the answer in a
// word that the subcycle kernel branches on: no synchronisation, the same
// launches either way, usable under stream capture.  On small grids an eager
// call runs the whole loop in one launch.
//
// The folded constants and half of the ping-pong state take the caller's
// pitch, so that everything the subcycle reads unchanged (ocean velocities,
// masses, areas, the first state) is read where the caller has it.
#include "evp_fast64.cuh"
#include "evp_residual.cuh"

namespace veris {

constexpr size_t AUTO_STATUS_BYTES = 256;   // the state check's word, and at +128 the loop's barrier count

struct AutoSpace {
    int *viol;
    Ctx<double> *ctx;
    FastConsts<double> c;
    double *sdU, *sdV;
    double *state[5];
};

// Carves the workspace; returns its size.
static size_t auto_layout(const Dims &d, const VerisParams &p, char *base, AutoSpace *a) {
    const size_t f2 = rup256((size_t)d.NX * d.ld * sizeof(double));
    const size_t fx = rup256((size_t)d.NX * sizeof(double)), fy = rup256((size_t)d.NY * sizeof(double));
    size_t off = 0;
    auto take = [&](size_t n) { char *q = base ? base + off : nullptr; off += n; return q; };
    auto field = [&](bool used) { return used ? reinterpret_cast<double *>(take(f2)) : nullptr; };
    const bool adapt = p.useAdaptiveEVP != 0, slip = p.noSlip == 0, basal = p.basalDragK2 != 0.0;
    a->viol = reinterpret_cast<int *>(take(AUTO_STATUS_BYTES));
    a->ctx = reinterpret_cast<Ctx<double> *>(take(rup256(sizeof(Ctx<double>))));
    FastConsts<double> &c = a->c;
    c = FastConsts<double>{};
    double **always[6] = {&c.rsqrA, &c.mf4, &c.cU, &c.cV, &c.hAW, &c.hAS};
    for (double **q : always) *q = field(true);
    double **constant[5] = {&c.Phh, &c.mUb, &c.mVb, &c.mUb1, &c.mVb1};
    for (double **q : constant) *q = field(!adapt);
    c.Ph = field(adapt);
    c.acf = field(adapt);
    c.bfac = field(basal);
    a->sdU = field(slip);
    a->sdV = field(slip);
    c.flags = reinterpret_cast<uint32_t *>(take(rup256((size_t)d.NX * d.ld * sizeof(uint32_t))));
    double **xs[4] = {&c.rdxU_x, &c.rdxVh_x, &c.dxV_x, &c.dxUh_x}, **ys[4] = {&c.rdyV_y, &c.rdyUh_y, &c.dyVh_y, &c.dyU_y};
    for (double **q : xs) *q = reinterpret_cast<double *>(take(fx));
    for (double **q : ys) *q = reinterpret_cast<double *>(take(fy));
    for (double *&q : a->state) q = reinterpret_cast<double *>(take(f2));
    return off;
}

// Folds the step's constants and checks the state.  Non-finite inputs take
// the plain tile too: it multiplies by the masks, so that a NaN on land
// spreads as in the reference, where the folded form selects.
__global__ void auto_prep_kernel(const __grid_constant__ Ctx<double> x, AutoSpace a) {
    const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 8 + threadIdx.y;
    const Dims &d = x.d;
    const VerisParams &p = x.p;
    const Fields<double> &f = x.f;
    if (blockIdx.x == 0 && blockIdx.y == 0) {
        const int *from = reinterpret_cast<const int *>(&x);
        for (int q = threadIdx.y * 32 + threadIdx.x; q < (int)(sizeof(x) / sizeof(int)); q += 256)
            reinterpret_cast<int *>(a.ctx)[q] = from[q];
    }
    if (i >= d.NX || j >= d.NY) return;
    const bool adapt = p.useAdaptiveEVP != 0, slip = p.noSlip == 0;
    const int64_t o = d.raw(i, j), oi = d.raw(i, 0), oj = d.raw(0, j);
    bool ok = f.k1AtC[o] == 0.0 && f.k2AtC[o] == 0.0 && f.k1AtZ[o] == 0.0 && f.k2AtZ[o] == 0.0;
    auto bit = [&](const double *m) {
        const double v = m[o];
        ok = ok && (v == 0.0 || v == 1.0);
        return v != 0.0;
    };
    auto num = [&](const double *q) {
        const double v = q[o];
        ok = ok && finite64(v);
        return v;
    };
    auto along = [&](const double *q, int64_t o0) {   // a grid length, equal to the one at o0
        const double v = q[o];
        ok = ok && v == q[o0] && finite64(v);
        return v;
    };
    const FastConsts<double> &c = a.c;
    const double rdt = p.recip_deltatDyn;
    const double mC = num(f.SeaIceMassC), mU = num(f.SeaIceMassU), mV = num(f.SeaIceMassV), fc = num(f.fCori);
    const double rrA = num(f.recip_rA);
    const double Ph = 0.5 * num(f.SeaIceStrength) * (1.0 + p.tensileStrFac);
    c.rsqrA[o] = rrA / (p.PlasDefCoeff * p.PlasDefCoeff);
    c.mf4[o] = 0.25 * mC * fc;
    c.cU[o] = mU * rdt * num(f.uIce) + num(f.WindForcingX);
    c.cV[o] = mV * rdt * num(f.vIce) + num(f.WindForcingY);
    c.hAW[o] = 0.5 * p.cosWat * num(f.AreaW);
    c.hAS[o] = 0.5 * p.cosWat * num(f.AreaS);
    ok = ok && finite64(f.sigma1[o]) && finite64(f.sigma2[o]) && finite64(f.sigma12[o]) && finite64(f.uOcean[o]) &&
         finite64(f.vOcean[o]) && finite64(f.rAz[o]) && finite64(f.recip_rAu[o]) && finite64(f.recip_rAv[o]);
    if (adapt) {   // veris/evp_solver.py:65-73, the state-only factor of alphaC
        c.Ph[o] = Ph;
        c.acf[o] = p.EVPcFac * rrA / (mC > 1e-4 ? mC : 1e-4);
    } else {
        const double bU = p.evpBeta * rdt, bU1 = bU + rdt;
        c.Phh[o] = Ph * (0.5 / p.evpAlpha);
        c.mUb[o] = bU * mU;
        c.mVb[o] = bU * mV;
        c.mUb1[o] = mU * bU1;
        c.mVb1[o] = mV * bU1;
    }
    if (p.basalDragK2 != 0.0) {
        const double A = num(f.Area), h = num(f.hIceMean), R = num(f.R_low);
        double b = 0.0;
        if (A > 0.01)
            b = p.basalDragK2 * log(exp(10.0 * (h - fabs(R) * A / p.basalDragK1)) + 1.0) * 0.1 *
                exp(-p.cBasalStar * (1.0 - A));
        ok = ok && finite64(b);
        c.bfac[o] = b;
    }
    uint32_t fl = 0;
    fl |= bit(f.iceMask) ? F_MC : 0;
    fl |= bit(f.maskInC) ? F_INC : 0;
    fl |= bit(f.iceMaskU) ? F_MU : 0;
    fl |= bit(f.maskInU) ? F_INU : 0;
    fl |= bit(f.iceMaskV) ? F_MV : 0;
    fl |= bit(f.maskInV) ? F_INV : 0;
    fl |= mU != 0.0 ? F_LMU : 0;
    fl |= mV != 0.0 ? F_LMV : 0;
    fl |= fc < 0.0 ? F_SOUTH | F_SNEG : 0;
    fl |= fc > 0.0 ? F_SPOS : 0;
    c.flags[o] = fl;
    if (slip) {   // veris/dynamics_routines.py:115-138, all but the speed
        const double cU = p.use_coastline ? num(f.Fu)
                                          : (2.0 - f.iceMaskU[d.at(i - 1, j)] - f.iceMaskU[d.at(i + 1, j)]) * f.iceMaskU[o];
        const double cV = p.use_coastline ? num(f.Fv)
                                          : (2.0 - f.iceMaskV[d.at(i, j - 1)] - f.iceMaskV[d.at(i, j + 1)]) * f.iceMaskV[o];
        a.sdU[o] = mU * p.sideDragCoeff * cU;
        a.sdV[o] = mV * p.sideDragCoeff * cV;
    }
    const double rdxU = along(f.recip_dxU, oi), rdxV = along(f.recip_dxV, oi);
    const double dxV = along(f.dxV, oi), dxU = along(f.dxU, oi);
    const double rdyV = along(f.recip_dyV, oj), rdyU = along(f.recip_dyU, oj);
    const double dyV = along(f.dyV, oj), dyU = along(f.dyU, oj);
    if (j == 0) {
        c.rdxU_x[i] = rdxU;
        c.rdxVh_x[i] = 0.5 * rdxV;
        c.dxV_x[i] = dxV;
        c.dxUh_x[i] = 0.5 * dxU;
    }
    if (i == 0) {
        c.rdyV_y[j] = rdyV;
        c.rdyUh_y[j] = 0.5 * rdyU;
        c.dyVh_y[j] = 0.5 * dyV;
        c.dyU_y[j] = dyU;
    }
    if (!ok) *a.viol = 1;
}

// Settings under which the folded form's algebra is the plain form's: no
// second-order boundary terms, replacement pressure on, and none of the
// limits in which one of the two divides by zero or takes a sign the other
// does not.
static bool folds(const VerisParams &p) {
    const bool adapt = p.useAdaptiveEVP != 0, slip = p.noSlip == 0, basal = p.basalDragK2 != 0.0;
    auto positive = [](double x) { return x > 0.0 && x < 1e300; };
    auto fin = [](double x) { return x > -1e300 && x < 1e300; };
    return (slip || !p.secondOrderBC) && p.pressReplFac == 1.0 && positive(p.deltaMin) &&
           positive(p.PlasDefCoeff) && positive(1.0 + p.tensileStrFac) && positive(p.evpAlpha) && fin(p.evpBeta) &&
           p.cDragMin >= 0.0 && fin(p.cDragMin) && p.waterIceDrag * p.rhoSea >= 0.0 &&
           p.waterIceDrag_south * p.rhoSea >= 0.0 && fin(p.waterIceDrag * p.rhoSea) &&
           fin(p.waterIceDrag_south * p.rhoSea) && positive(p.recip_deltatDyn) && fin(p.cosWat) && fin(p.sinWat) &&
           (!adapt || (positive(p.aEVPalphaMin) && p.EVPcFac >= 0.0 && fin(p.EVPcFac))) &&
           (!slip || (positive(p.sideDragU0) && fin(p.sideDragCoeff))) &&
           (!basal || (p.basalDragU0 != 0.0 && fin(p.basalDragU0) && p.basalDragK1 != 0.0 && fin(p.basalDragK1) &&
                       fin(p.basalDragK2) && fin(p.cBasalStar)));
}

// Units of 24 rows as in the engine's loop; with adaptive or side terms the
// 16-row tile, whose arrays still fit three CTAs per SM.
template <bool B, bool R>
static int auto_launch(bool adapt, bool slip, const Dims &d, const HaloFill &h, const FastConsts<double> &c,
                       const F64Scalars &k, const FastIO<double> &io, cudaStream_t st, const F64Auto &a) {
    if (adapt)
        return slip ? launch64<16, B, R, false, true, true, true>(d, d.ld, h, c, k, io, st, a)
                    : launch64<16, B, R, false, true, false, true>(d, d.ld, h, c, k, io, st, a);
    return slip ? launch64<16, B, R, false, false, true, true>(d, d.ld, h, c, k, io, st, a)
                : launch64<24, B, R, false, false, false, true>(d, d.ld, h, c, k, io, st, a);
}

// the whole loop in one launch, on the grids that take it
template <bool B, bool R>
static int auto_loop_launch(bool adapt, bool slip, const Dims &d, const HaloFill &h, const FastConsts<double> &c,
                            const F64Scalars &k, const F64Loop &l, cudaStream_t st, const F64Auto &a) {
    if (adapt)
        return slip ? launch64_loop<B, R, true, true>(d, d.ld, h, c, k, l, st, a)
                    : launch64_loop<B, R, true, false>(d, d.ld, h, c, k, l, st, a);
    return slip ? launch64_loop<B, R, false, true>(d, d.ld, h, c, k, l, st, a)
                : launch64_loop<B, R, false, false>(d, d.ld, h, c, k, l, st, a);
}

// where a loop with residual diagnostics keeps alphaC and the partial sums
struct AutoResidual {
    double *aC, *partial;
};

// the prep and n subcycles, the last into outs; res: the residuals' partial
// sums after each
static int auto_loop(const Dims &d, const VerisParams *p, const VerisFieldsF64 *vs, AutoSpace &a, int n, double *u,
                     double *v, double *s1, double *s2, double *s12, const AutoResidual *res, cudaStream_t st) {
    if (cudaMemsetAsync(a.viol, 0, AUTO_STATUS_BYTES, st) != cudaSuccess) return VERIS_ERR_LAUNCH;
    Ctx<double> x;
    x.f = *reinterpret_cast<const Fields<double> *>(vs);
    x.d = d;
    x.p = *p;
    FastConsts<double> &c = a.c;
    c.rAz = const_cast<double *>(x.f.rAz);
    c.rrAu = const_cast<double *>(x.f.recip_rAu);
    c.rrAv = const_cast<double *>(x.f.recip_rAv);
    c.uOc = const_cast<double *>(x.f.uOcean);
    c.vOc = const_cast<double *>(x.f.vOcean);
    c.AW = const_cast<double *>(x.f.AreaW);
    c.AS = const_cast<double *>(x.f.AreaS);
    c.mU = const_cast<double *>(x.f.SeaIceMassU);
    c.mV = const_cast<double *>(x.f.SeaIceMassV);
    dim3 g2((d.NY + 31) / 32, (d.NX + 7) / 8);
    auto_prep_kernel<<<g2, dim3(32, 8), 0, st>>>(x, a);
    int stt = launch_status();
    if (stt != VERIS_OK) return stt;
    const F64Scalars k = f64_scalars(fast_scalars<double>(*p), p->sideDragU0);
    const HaloFill h = halo_fill_of(*p);
    const F64Auto aa{a.viol, a.ctx, a.sdU, a.sdV};
    const bool adapt = p->useAdaptiveEVP != 0, slip = p->noSlip == 0, basal = p->basalDragK2 != 0.0,
               turn = p->sinWat != 0.0;
    double *const outs[5] = {u, v, s1, s2, s12};
    const double *cur[5] = {x.f.uIce, x.f.vIce, x.f.sigma1, x.f.sigma2, x.f.sigma12};
    // a graph has no host time per launch to save
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const bool eager = cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    if (!eager) cudaGetLastError();
    if (!res && eager) {
        F64Loop l;
        for (int q = 0; q < 5; ++q) {
            l.in[q] = cur[q];
            l.even[q] = (n - 1) % 2 ? a.state[q] : outs[q];
            l.odd[q] = (n - 1) % 2 ? outs[q] : a.state[q];
            l.out[q] = outs[q];
        }
        l.ldo = d.ld;
        l.n = n;
        l.arrived = reinterpret_cast<unsigned *>(a.viol) + 32;
        stt = basal ? (turn ? auto_loop_launch<true, true>(adapt, slip, d, h, c, k, l, st, aa)
                            : auto_loop_launch<true, false>(adapt, slip, d, h, c, k, l, st, aa))
                    : (turn ? auto_loop_launch<false, true>(adapt, slip, d, h, c, k, l, st, aa)
                            : auto_loop_launch<false, false>(adapt, slip, d, h, c, k, l, st, aa));
        if (stt == VERIS_OK) return stt;   // else one launch per subcycle
    }
    for (int it = 0; it < n; ++it) {
        double *const *dst = (n - 1 - it) % 2 ? a.state : outs;
        FastIO<double> io{cur[0], cur[1], cur[2], cur[3], cur[4], dst[0], dst[1], dst[2], dst[3], dst[4], d.ld};
        if (res && adapt) io.aCo = res->aC;
        stt = basal ? (turn ? auto_launch<true, true>(adapt, slip, d, h, c, k, io, st, aa)
                            : auto_launch<true, false>(adapt, slip, d, h, c, k, io, st, aa))
                    : (turn ? auto_launch<false, true>(adapt, slip, d, h, c, k, io, st, aa)
                            : auto_launch<false, false>(adapt, slip, d, h, c, k, io, st, aa));
        if (stt != VERIS_OK) return stt;
        if (res) {
            const ResIO<double> r{cur[0], cur[1], cur[2], cur[3], cur[4], dst[0], dst[1], dst[2], dst[3], dst[4],
                                  vs->iceMask, vs->iceMaskU, vs->iceMaskV, adapt ? res->aC : nullptr, p->evpAlpha,
                                  p->evpBeta};
            stt = residual_partial<double>(d, r, res->partial + (int64_t)it * 2 * res_blocks(d), st);
            if (stt != VERIS_OK) return stt;
        }
        for (int q = 0; q < 5; ++q) cur[q] = dst[q];
    }
    return VERIS_OK;
}

}  // namespace veris

using namespace veris;

extern "C" {

size_t veris_evp_auto_workspace_bytes(const VerisGrid *g, const VerisParams *p) {
    Dims d;
    if (!p || check_grid(g, &d) != VERIS_OK) return 0;
    if (!folds(*p)) return veris_evp_workspace_bytes(g, 8);
    AutoSpace a;
    return auto_layout(d, *p, nullptr, &a);
}

int veris_evp_auto_solver_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, int32_t n,
                              double *u, double *v, double *s1, double *s2, double *s12, void *ws, size_t wsb,
                              veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && u && v && s1 && s2 && s12, VERIS_ERR_ARG);
    VERIS_REQUIRE(n >= 0, VERIS_ERR_ARG);
    if (n == 0 || !folds(*p)) return veris_evp_solver_f64(g, p, vs, n, u, v, s1, s2, s12, ws, wsb, s);
    AutoSpace a;
    VERIS_REQUIRE(ws && wsb >= auto_layout(d, *p, nullptr, &a), VERIS_ERR_WORKSPACE);
    auto_layout(d, *p, static_cast<char *>(ws), &a);
    return auto_loop(d, p, vs, a, n, u, v, s1, s2, s12, nullptr, (cudaStream_t)s);
}

size_t veris_evp_auto_residual_workspace_bytes(const VerisGrid *g, const VerisParams *p, int32_t n) {
    Dims d;
    if (!p || n < 0 || check_grid(g, &d) != VERIS_OK) return 0;
    if (!folds(*p)) return veris_evp_residual_workspace_bytes(g, 8, n);
    AutoSpace a;
    return auto_layout(d, *p, nullptr, &a) + rup256((size_t)d.NX * d.ld * sizeof(double)) +
           (size_t)n * 2 * res_blocks(d) * sizeof(double);
}

int veris_evp_auto_residual_solver_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, int32_t n,
                                       double *u, double *v, double *s1, double *s2, double *s12, double *resU,
                                       double *resSig, void *ws, size_t wsb, veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && u && v && s1 && s2 && s12, VERIS_ERR_ARG);
    VERIS_REQUIRE(n >= 0, VERIS_ERR_ARG);
    if (n == 0 || !folds(*p))
        return veris_evp_residual_solver_f64(g, p, vs, n, u, v, s1, s2, s12, resU, resSig, ws, wsb, s);
    VERIS_REQUIRE(resU && resSig, VERIS_ERR_ARG);
    VERIS_REQUIRE(ws && wsb >= veris_evp_auto_residual_workspace_bytes(g, p, n), VERIS_ERR_WORKSPACE);
    AutoSpace a;
    char *base = static_cast<char *>(ws);
    base += auto_layout(d, *p, base, &a);
    AutoResidual res;
    res.aC = reinterpret_cast<double *>(base);
    res.partial = reinterpret_cast<double *>(base + rup256((size_t)d.NX * d.ld * sizeof(double)));
    const int stt = auto_loop(d, p, vs, a, n, u, v, s1, s2, s12, &res, (cudaStream_t)s);
    if (stt != VERIS_OK) return stt;
    return residual_finish(d, res.partial, n, resU, resSig, (cudaStream_t)s);
}

}  // extern "C"
