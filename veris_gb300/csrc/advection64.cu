// Float64 flux-limited advection (veris/advection.py:15-175) in two launches,
// zonal and meridional, each a flux and its update in one pass.
//
// Bound by the float64 pipe.  The separate passes (transport, flux, update,
// flux, update: advection.cu) evaluated each limiter with an IEEE division and
// every comparison, sign and 0/1 mask on that pipe, 35 operations per flux of
// every cell, and formed the Courant number and the slopes anew for each
// field.  Here the superbee limiter decides on the integer pipe which of its
// branches holds, so that only slope ratios in (0, 1/2) and (1, 2) are divided,
// masks of 1 are not multiplied, the transport, Courant number and update
// factor serve all fields, a slope is formed once, and warps without ice (four
// zero values around the face in every field) skip the flux.
// 1444 x 724, three fields: 549 us in five launches; here 68 and 71 us (float64
// pipe 68 and 73 % busy; 79 and 76 us with the divisions on it).
//
// Face i of axis 0 (j of axis 1) takes field values f[i-2 .. i+1]; the fluxes
// vanish outside [2, N-2] and the halo fill that the reference applies to them
// makes a halo face the image of its interior source, which is what is
// evaluated there.
#include "advection64.cuh"
#include "f64math.cuh"
#include "stencil.cuh"

namespace veris {

namespace {

constexpr int WARPS = 4;

__device__ __forceinline__ bool is_one(double x) { return bits_of(x) == 0x3ff0000000000000ULL; }
__device__ __forceinline__ double masked(double x, double m) { return is_one(m) ? x : x * m; }
__device__ __forceinline__ double mask2(double a, double b) { return is_one(a) ? b : a * b; }
__device__ __forceinline__ unsigned long long abs_bits(double x) { return bits_of(x) & 0x7fffffffffffffffULL; }
__device__ __forceinline__ double abs64(double x) { return __longlong_as_double((long long)abs_bits(x)); }

// limited flux (veris/advection.py:107-126, superbee :170-175) from the values
// fm, f0 beside the face, the slopes there, half the transport and the Courant
// number; CrMax at least 2, beyond which superbee is constant
__device__ __forceinline__ double limited_flux64(double fm, double f0, double Rjm, double Rj, double Rjp, double th,
                                                 double cfl) {
    const double cr = is_pos(th) ? Rjm : Rjp;
    const unsigned long long a = abs_bits(Rj), c = abs_bits(cr), inf = 0x7ff0000000000000ULL;
    double w = 1.0;   // (1 - phi) + cfl phi
    // phi > 0: slopes of one sign, neither zero nor NaN
    if (((bits_of(Rj) ^ bits_of(cr)) >> 63) == 0 && a != 0 && c != 0 && a <= inf && c <= inf) {
        const double r = __longlong_as_double((long long)a), q = __longlong_as_double((long long)c);
        // halves and doubles by the exponent (exact; below 2^-1021 by the pipe)
        const bool tiny = a < (2ULL << 52) || c < (2ULL << 52);
        const unsigned long long c2 = tiny ? abs_bits(2.0 * q) : c + (c < inf ? 1ULL << 52 : 0),
                                 a2 = tiny ? abs_bits(2.0 * r) : a + (a < inf ? 1ULL << 52 : 0);
        double phi;
        if (c >= a2) phi = 2.0;
        else if (c <= a && c2 >= a) phi = 1.0;
        else {
            phi = div_lane(q, r);
            if (c < a) phi = phi + phi;
        }
        w = fma(cfl, phi, 1.0 - phi);
    }
    return fma(-abs64(th) * Rj, w, th * (f0 + fm));
}

__device__ __forceinline__ bool any_bits(double a, double b, double c, double d) {
    return ((bits_of(a) | bits_of(b) | bits_of(c) | bits_of(d)) << 1) != 0;
}

// f1 = f - dt/rA maskInC (F(i+1) - F(i)): one warp per 32 columns walks down
// H rows; the slopes and the flux of the row above stay in registers.  Seven
// CTAs per SM (73 registers) hold all walks of 1444 x 724 at once: 79 us; with
// 84 registers the last walks ran alone, 92 us; eight CTAs spill, 81 us.
template <int NF>
__global__ void __launch_bounds__(WARPS * 32, 7) zonal_kernel(const __grid_constant__ Ctx<double> c, HaloFill h,
                                                           Adv64IO io, int nstrips, int H) {
    const Dims &d = c.d;
    const Fields<double> &f = c.f;
    // the warps of a CTA take walks far apart, so that ice (some strips of
    // columns) and open water share every SM
    const int lane = threadIdx.x & 31, w = blockIdx.x + (threadIdx.x >> 5) * gridDim.x;
    const int i0 = (w / nstrips) * H;
    if (i0 >= d.NX) return;
    const int jl = (w % nstrips) * 32 + lane;
    const bool live = jl < d.NY;
    const int j = live ? jl : d.NY - 1;
    // the column whose fluxes this column's are (y halo of a doubly periodic fill)
    const int jf = h.y_fill && in_yhalo(d, h.oly, j) ? (j < h.oly ? j + d.ny : j - d.ny) : j;
    const int i1 = min(i0 + H, d.NX);
    auto m = [&](int64_t q) { return mask2(__ldg(f.iceMaskU + q), __ldg(f.maskInU + q)); };
    double a0[NF], a1[NF], Rm[NF], R0[NF], F[NF];   // f at s-1 and s, slopes at s-1 and s, the flux of the row before
    int have = -9;                                   // the face s that the window stands at
    for (int i = i0; i <= i1; ++i) {
        // face i (the one below the last row included), its source row s
        int s = i == d.NX ? 0 : i;
        if (h.x_fill && in_xhalo(d, h.olx, s)) s = s < h.olx ? s + d.nx : s - d.nx;
        double Fn[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) Fn[q] = 0.0;
        if (s >= 2 && s <= d.NX - 2) {
            const int64_t o = d.raw(s, jf);
            const int64_t L = d.ld;
            if (s != have + 1) {
                const double mm = m(o - L), m0 = m(o);
#pragma unroll
                for (int q = 0; q < NF; ++q) {
                    const double b = __ldg(io.field[q] + o - 2 * L);
                    a0[q] = __ldg(io.field[q] + o - L);
                    a1[q] = __ldg(io.field[q] + o);
                    Rm[q] = masked(a0[q] - b, mm);
                    R0[q] = masked(a1[q] - a0[q], m0);
                }
            }
            have = s;
            const double u = __ldg(f.uIce + o);
            const double t = 0.5 * u * mask2(__ldg(f.iceMaskU + o), __ldg(f.dyG + o));
            const double mp = m(o + L);
            double an[NF];
            bool some = !finite64(u);
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                an[q] = __ldg(io.field[q] + o + L);
                some = some || any_bits(a0[q], a1[q], an[q], Rm[q]);
            }
            if (__any_sync(0xffffffffu, some)) {
                const double cfl = abs64(u * c.p.deltatTherm * __ldg(f.recip_dxC + o));
#pragma unroll
                for (int q = 0; q < NF; ++q) {
                    const double Rp = masked(an[q] - a1[q], mp);
                    Fn[q] = limited_flux64(a0[q], a1[q], Rm[q], R0[q], Rp, t, cfl);
                    Rm[q] = R0[q];
                    R0[q] = Rp;
                }
            } else {
#pragma unroll
                for (int q = 0; q < NF; ++q) {
                    Rm[q] = R0[q];
                    R0[q] = 0.0;   // all values are zero
                }
            }
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                a0[q] = a1[q];
                a1[q] = an[q];
            }
        }
        if (i > i0 && live) {
            const int64_t o = d.raw(i - 1, j);
            bool some = false;
#pragma unroll
            for (int q = 0; q < NF; ++q) some = some || any_bits(F[q], Fn[q], 0.0, 0.0);
            double k = 0.0;
            if (some) k = c.p.deltatTherm * masked(__ldg(f.recip_rA + o), __ldg(f.maskInC + o));
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                double v = __ldg(io.field[q] + o);
                if (some) v = fma(-k, Fn[q] - F[q], v);
                io.f1[q][o] = v;
            }
        }
#pragma unroll
        for (int q = 0; q < NF; ++q) F[q] = Fn[q];
    }
}

// out = (f1 - dt/rA maskInC (G(j+1) - G(j))) iceMask: a CTA takes one row of
// COLS columns, slopes and fluxes through shared memory.  Reads the fields
// from f1 only, so out may be the fields themselves.
constexpr int COLS = 128;
template <int NF>
__global__ void __launch_bounds__(COLS) meridional_kernel(const __grid_constant__ Ctx<double> c, HaloFill h,
                                                          Adv64IO io) {
    const Dims &d = c.d;
    const Fields<double> &f = c.f;
    __shared__ double sf[NF][COLS + 4], sR[NF][COLS + 4], sG[NF][COLS + 1];
    const int i = blockIdx.y, j0 = blockIdx.x * COLS, tid = threadIdx.x;
    // the row whose fluxes this row's are (x halo)
    const int r = h.x_fill && in_xhalo(d, h.olx, i) ? (i < h.olx ? i + d.nx : i - d.nx) : i;
    auto m = [&](int64_t q) { return mask2(__ldg(f.iceMaskV + q), __ldg(f.maskInV + q)); };
    // columns j0-2 .. j0+COLS+1; faces outside [2, NY-2] are not evaluated
    for (int q = 0; q < NF; ++q)
        for (int k = tid; k < COLS + 4; k += COLS) {
            const int j = j0 - 2 + k;
            sf[q][k] = j >= 0 && j < d.NY ? __ldg(io.f1[q] + d.raw(r, j)) : 0.0;
        }
    __syncthreads();
    for (int k = tid; k < COLS + 3; k += COLS) {   // slope at the face of column j0-1+k
        const int j = j0 - 1 + k;
        const bool in = j >= 1 && j < d.NY;
        const double mk = in ? m(d.raw(r, j)) : 0.0;
#pragma unroll
        for (int q = 0; q < NF; ++q) sR[q][k] = in ? masked(sf[q][k + 1] - sf[q][k], mk) : 0.0;
    }
    __syncthreads();
    for (int k = tid; k < COLS + 1; k += COLS) {
        int j = j0 + k;
        if (j > d.NY) break;
        if (j == d.NY) j = 0;
        double G[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) G[q] = 0.0;
        const bool image = h.y_fill && in_yhalo(d, h.oly, j);
        if (image) j = j < h.oly ? j + d.ny : j - d.ny;
        if (j >= 2 && j <= d.NY - 2) {
            const int64_t o = d.raw(r, j);
            const double v = __ldg(f.vIce + o);
            bool some = !finite64(v);
            if (!image) {
#pragma unroll
                for (int q = 0; q < NF; ++q)
                    some = some || any_bits(sf[q][k], sf[q][k + 1], sf[q][k + 2], sf[q][k + 3]);
            }
            if (some || image) {
                const double t = 0.5 * v * mask2(__ldg(f.iceMaskV + o), __ldg(f.dxG + o));
                const double cfl = abs64(v * c.p.deltatTherm * __ldg(f.recip_dyC + o));
#pragma unroll
                for (int q = 0; q < NF; ++q) {
                    double fm, f0, Rm, R0, Rp;
                    if (image) {
                        const double *p = io.f1[q] + o;
                        fm = __ldg(p - 1);
                        f0 = __ldg(p);
                        Rm = masked(fm - __ldg(p - 2), m(o - 1));
                        R0 = masked(f0 - fm, m(o));
                        Rp = masked(__ldg(p + 1) - f0, m(o + 1));
                    } else {
                        fm = sf[q][k + 1];
                        f0 = sf[q][k + 2];
                        Rm = sR[q][k];
                        R0 = sR[q][k + 1];
                        Rp = sR[q][k + 2];
                    }
                    G[q] = limited_flux64(fm, f0, Rm, R0, Rp, t, cfl);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NF; ++q) sG[q][k] = G[q];
    }
    __syncthreads();
    const int j = j0 + tid;
    if (j >= d.NY) return;
    const int64_t o = d.raw(i, j);
    const double mask = __ldg(f.iceMask + o);
    bool some = false;
#pragma unroll
    for (int q = 0; q < NF; ++q) some = some || any_bits(sG[q][tid], sG[q][tid + 1], 0.0, 0.0);
    double k = 0.0;
    if (some) k = c.p.deltatTherm * masked(__ldg(f.recip_rA + o), __ldg(f.maskInC + o));
#pragma unroll
    for (int q = 0; q < NF; ++q) {
        double v = r == i ? sf[q][tid + 2] : __ldg(io.f1[q] + o);
        if (some) v = fma(-k, sG[q][tid + 1] - sG[q][tid], v);
        io.out[q][o] = masked(v, mask);
    }
}

template <int NF>
int launch(const Ctx<double> &c, const HaloFill &h, const Adv64IO &io, cudaStream_t st) {
    const Dims &d = c.d;
    const int nstrips = (d.NY + 31) / 32;
    // eight rows a walk (one flux of nine is formed twice), fewer where the
    // walks would leave warp slots of the GPU empty
    int H = 8;
    const int sms = sm_count();
    while (H > 1 && (int64_t)nstrips * ((d.NX + H - 1) / H) < (int64_t)sms * 16) H /= 2;
    const int walks = nstrips * ((d.NX + H - 1) / H);
    zonal_kernel<NF><<<(walks + WARPS - 1) / WARPS, WARPS * 32, 0, st>>>(c, h, io, nstrips, H);
    int stt = launch_status();
    if (stt != VERIS_OK) return stt;
    meridional_kernel<NF><<<dim3((d.NY + COLS - 1) / COLS, d.NX), COLS, 0, st>>>(c, h, io);
    return launch_status();
}

}  // namespace

bool advect64_covers(const VerisParams &p, const Dims &d) { return p.CrMax >= 2.0 && d.NX <= 65535; }

int advect64(const Ctx<double> &c, const HaloFill &h, const Adv64IO &io, int nf, cudaStream_t st) {
    return nf == 1 ? launch<1>(c, h, io, st) : launch<3>(c, h, io, st);
}

}  // namespace veris
