// The mEVP subcycle loop (veris/evp_solver.py:21-319), plain form: one tiled
// kernel per subcycle (the tile is in evp_plain.cuh).  Inputs and outputs
// alternate between the caller's output arrays and the workspace (ping-pong),
// so no CTA reads a value another CTA of the same launch writes.
#include <mutex>

#include "evp_plain.cuh"
#include "evp_residual.cuh"
#include "tile_units.cuh"

namespace veris {

constexpr int PLAIN_ROWS = 32;   // rows of a tile at most

template <class T, bool ADAPT, bool SIDE, bool BASAL>
__global__ void __launch_bounds__(EVP_THREADS, 2)
evp_subcycle_kernel(Ctx<T> c, HaloFill h, EvpIO<T> io, TileUnits w) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int i0, ti, j0;
    w.unit(blockIdx.x, c.d.NX, i0, ti, j0);
    chain_wait();
    plain_tile<T, PLAIN_ROWS, ADAPT, SIDE, BASAL>(smem_raw, c, h, io, i0, ti, j0);
}

template <class T, bool A, bool Sd, bool B>
static int launch_subcycle(const Ctx<T> &c, const HaloFill &h, const EvpIO<T> &io, cudaStream_t st) {
    auto kern = evp_subcycle_kernel<T, A, Sd, B>;
    const size_t sm = PlainSmem<T, PLAIN_ROWS, A, Sd, B>::bytes();
    static std::atomic<bool> configured[MAX_DEVICES];
    if (!smem_configured(configured, kern, (int)sm)) return VERIS_ERR_LAUNCH;
    static std::atomic<int> resident[MAX_DEVICES];
    const int slots = cta_slots(resident, kern, EVP_THREADS, sm);
    if (slots <= 0) return VERIS_ERR_LAUNCH;
    const TileUnits w = tile_units(c.d, PLAIN_ROWS, slots);
    return launch_chained(kern, dim3(w.count), dim3(EVP_THREADS), sm, st, c, h, io, w);
}

template <class T>
static int dispatch_subcycle(const Ctx<T> &c, const HaloFill &h, const EvpIO<T> &io, cudaStream_t st) {
    const bool A = c.p.useAdaptiveEVP != 0, Sd = c.p.noSlip == 0, B = c.p.basalDragK2 != 0.0;
    if (A) {
        if (Sd) return B ? launch_subcycle<T, true, true, true>(c, h, io, st) : launch_subcycle<T, true, true, false>(c, h, io, st);
        return B ? launch_subcycle<T, true, false, true>(c, h, io, st) : launch_subcycle<T, true, false, false>(c, h, io, st);
    }
    if (Sd) return B ? launch_subcycle<T, false, true, true>(c, h, io, st) : launch_subcycle<T, false, true, false>(c, h, io, st);
    return B ? launch_subcycle<T, false, false, true>(c, h, io, st) : launch_subcycle<T, false, false, false>(c, h, io, st);
}

static size_t field_bytes(const Dims &d, size_t elem) { return (size_t)d.NX * (size_t)d.ld * elem; }

static size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

template <class T>
static int evp_solver(const VerisGrid *g, const VerisParams *p, const Fields<T> *vs, int n, T *u, T *v,
                      T *s1, T *s2, T *s12, void *ws, size_t ws_bytes, veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && u && v && s1 && s2 && s12, VERIS_ERR_ARG);
    VERIS_REQUIRE(n >= 0, VERIS_ERR_ARG);
    cudaStream_t st = (cudaStream_t)s;
    const size_t fb = round_up(field_bytes(d, sizeof(T)), 256);
    if (n == 0) {
        const T *src[5] = {vs->uIce, vs->vIce, vs->sigma1, vs->sigma2, vs->sigma12};
        T *dst[5] = {u, v, s1, s2, s12};
        for (int q = 0; q < 5; ++q)
            if (cudaMemcpyAsync(dst[q], src[q], field_bytes(d, sizeof(T)), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
                return VERIS_ERR_LAUNCH;
        return VERIS_OK;
    }
    if (n > 1) VERIS_REQUIRE(ws && ws_bytes >= 5 * fb, VERIS_ERR_WORKSPACE);
    Ctx<T> c;
    c.f = *vs;
    c.d = d;
    c.p = *p;
    const HaloFill h = halo_fill_of(*p);
    T *buf[2][5] = {{u, v, s1, s2, s12}, {nullptr, nullptr, nullptr, nullptr, nullptr}};
    if (n > 1)
        for (int q = 0; q < 5; ++q) buf[1][q] = reinterpret_cast<T *>(static_cast<char *>(ws) + q * fb);
    const T *cur[5] = {vs->uIce, vs->vIce, vs->sigma1, vs->sigma2, vs->sigma12};
    for (int it = 0; it < n; ++it) {
        T **dst = buf[(n - 1 - it) % 2];
        EvpIO<T> io{cur[0], cur[1], cur[2], cur[3], cur[4], dst[0], dst[1], dst[2], dst[3], dst[4],
                    vs->uIce, vs->vIce};
        const int stt = dispatch_subcycle<T>(c, h, io, st);
        if (stt != VERIS_OK) return stt;
        for (int q = 0; q < 5; ++q) cur[q] = dst[q];
    }
    return VERIS_OK;
}

// ---------------------------------------------------------------------------
// Residual diagnostics (veris/evp_solver.py:193-234, computeEvpResidual), as
// that branch means them (it reads names it never binds): after subcycle k,
// over the interior points,
//   resSig[k] = sum (d sig11 alphaC iceMask)^2 + (d sig22 alphaC iceMask)^2 + (d sigma12 alphaZ)^2
//   resU[k]   = sum (iceMaskU d uIce betaU)^2 + (iceMaskV d vIce betaV)^2
// with sig11, sig22 = (sigma1 +- sigma2) / 2 and d the change over the
// subcycle.  The ping-pong keeps the state before the subcycle intact, so the
// residual kernel reads both states directly.  The sums are in float64 and
// deterministic: a fixed grid (a function of the interior size only), warp
// shuffles and one partial pair per block, then one block per subcycle adds
// the partials in index order.

__device__ __forceinline__ double warp_sum(double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

template <class T>
__global__ void __launch_bounds__(RES_THREADS) evp_residual_kernel(Dims d, ResIO<T> r, double *partial) {
    __shared__ double red[2][RES_THREADS / 32];
    const int ox = (d.NX - d.nx) / 2, oy = (d.NY - d.ny) / 2;
    double su = 0.0, ss = 0.0;
    for (int row = blockIdx.x; row < d.nx; row += gridDim.x)
    for (int col = threadIdx.x; col < d.ny; col += RES_THREADS) {
        const int64_t o = d.raw(ox + row, oy + col);
        // (d sig11)^2 + (d sig22)^2 = 0.5 ((d sigma1)^2 + (d sigma2)^2); with
        // constant alpha and beta their squares multiply the block sums instead
        const double d1 = (double)r.s11[o] - (double)r.s10[o], d2 = (double)r.s21[o] - (double)r.s20[o];
        const double d12 = (double)r.s121[o] - (double)r.s120[o];
        const double du = (double)r.mU[o] * ((double)r.u1[o] - (double)r.u0[o]);
        const double dv = (double)r.mV[o] * ((double)r.v1[o] - (double)r.v0[o]);
        const double mC = r.mC[o];
        const double c2 = fma(d1, d1, d2 * d2) * (0.5 * (mC * mC));
        if (r.aC) {
            const double a0 = r.aC[o], aw = r.aC[o - d.ld], as = r.aC[o - 1], asw = r.aC[o - d.ld - 1];
            const double aZ = 0.5 * (0.5 * (a0 + as) + 0.5 * (aw + asw));
            const double bU = 0.5 * (a0 + aw), bV = 0.5 * (a0 + as);
            ss += c2 * (a0 * a0) + (d12 * aZ) * (d12 * aZ);
            su += (du * bU) * (du * bU) + (dv * bV) * (dv * bV);
        } else {
            ss += fma(d12, d12, c2);
            su += fma(du, du, dv * dv);
        }
    }
    if (!r.aC) {
        su *= r.beta * r.beta;
        ss *= r.alpha * r.alpha;
    }
    su = warp_sum(su);
    ss = warp_sum(ss);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = su;
        red[1][w] = ss;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        su = threadIdx.x < RES_THREADS / 32 ? red[0][threadIdx.x] : 0.0;
        ss = threadIdx.x < RES_THREADS / 32 ? red[1][threadIdx.x] : 0.0;
        su = warp_sum(su);
        ss = warp_sum(ss);
        if (threadIdx.x == 0) {
            partial[2 * blockIdx.x] = su;
            partial[2 * blockIdx.x + 1] = ss;
        }
    }
}

// one block per subcycle: the partials of that subcycle in index order
__global__ void __launch_bounds__(RES_THREADS) evp_residual_finish_kernel(const double *partial, int nblk,
                                                                          double *resU, double *resSig) {
    __shared__ double red[2][RES_THREADS / 32];
    const double *pk = partial + (int64_t)blockIdx.x * 2 * nblk;
    double su = 0.0, ss = 0.0;
    for (int b = threadIdx.x; b < nblk; b += RES_THREADS) {
        su += pk[2 * b];
        ss += pk[2 * b + 1];
    }
    su = warp_sum(su);
    ss = warp_sum(ss);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = su;
        red[1][w] = ss;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        su = threadIdx.x < RES_THREADS / 32 ? red[0][threadIdx.x] : 0.0;
        ss = threadIdx.x < RES_THREADS / 32 ? red[1][threadIdx.x] : 0.0;
        su = warp_sum(su);
        ss = warp_sum(ss);
        if (threadIdx.x == 0) {
            resU[blockIdx.x] = su;
            resSig[blockIdx.x] = ss;
        }
    }
}

template <class T>
int residual_partial(const Dims &d, const ResIO<T> &r, double *partial, cudaStream_t st) {
    evp_residual_kernel<T><<<res_blocks(d), RES_THREADS, 0, st>>>(d, r, partial);
    return launch_status();
}
template int residual_partial<double>(const Dims &, const ResIO<double> &, double *, cudaStream_t);

int residual_finish(const Dims &d, const double *partial, int n, double *resU, double *resSig, cudaStream_t st) {
    evp_residual_finish_kernel<<<n, RES_THREADS, 0, st>>>(partial, res_blocks(d), resU, resSig);
    return launch_status();
}

static size_t residual_workspace_bytes(const Dims &d, size_t elem, int n) {
    return 6 * round_up(field_bytes(d, elem), 256) + (size_t)(n > 0 ? n : 0) * 2 * res_blocks(d) * sizeof(double);
}

template <class T>
static int evp_residual_solver(const VerisGrid *g, const VerisParams *p, const Fields<T> *vs, int n, T *u, T *v,
                               T *s1, T *s2, T *s12, double *resU, double *resSig, void *ws, size_t ws_bytes,
                               veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    VERIS_REQUIRE(p && vs && u && v && s1 && s2 && s12, VERIS_ERR_ARG);
    VERIS_REQUIRE(n >= 0, VERIS_ERR_ARG);
    if (n == 0) return evp_solver<T>(g, p, vs, 0, u, v, s1, s2, s12, ws, ws_bytes, s);
    VERIS_REQUIRE(resU && resSig, VERIS_ERR_ARG);
    VERIS_REQUIRE(ws && ws_bytes >= residual_workspace_bytes(d, sizeof(T), n), VERIS_ERR_WORKSPACE);
    cudaStream_t st = (cudaStream_t)s;
    const size_t fb = round_up(field_bytes(d, sizeof(T)), 256);
    Ctx<T> c;
    c.f = *vs;
    c.d = d;
    c.p = *p;
    const HaloFill h = halo_fill_of(*p);
    const bool adapt = p->useAdaptiveEVP != 0;
    char *base = static_cast<char *>(ws);
    T *buf[2][5] = {{u, v, s1, s2, s12}, {nullptr, nullptr, nullptr, nullptr, nullptr}};
    for (int q = 0; q < 5; ++q) buf[1][q] = reinterpret_cast<T *>(base + q * fb);
    T *aC = reinterpret_cast<T *>(base + 5 * fb);
    double *partial = reinterpret_cast<double *>(base + 6 * fb);
    const int nblk = res_blocks(d);
    const T *cur[5] = {vs->uIce, vs->vIce, vs->sigma1, vs->sigma2, vs->sigma12};
    for (int it = 0; it < n; ++it) {
        T **dst = buf[(n - 1 - it) % 2];
        EvpIO<T> io{cur[0], cur[1], cur[2], cur[3], cur[4], dst[0], dst[1], dst[2], dst[3], dst[4],
                    vs->uIce, vs->vIce, adapt ? aC : nullptr};
        int stt = dispatch_subcycle<T>(c, h, io, st);
        if (stt != VERIS_OK) return stt;
        ResIO<T> r{cur[0], cur[1], cur[2], cur[3], cur[4], dst[0], dst[1], dst[2], dst[3], dst[4],
                   vs->iceMask, vs->iceMaskU, vs->iceMaskV, adapt ? aC : nullptr, p->evpAlpha, p->evpBeta};
        stt = residual_partial<T>(d, r, partial + (int64_t)it * 2 * nblk, st);
        if (stt != VERIS_OK) return stt;
        for (int q = 0; q < 5; ++q) cur[q] = dst[q];
    }
    return residual_finish(d, partial, n, resU, resSig, st);
}

}  // namespace veris

using namespace veris;

extern "C" {

size_t veris_evp_residual_workspace_bytes(const VerisGrid *g, int32_t elem_size, int32_t n_subcycles) {
    Dims d;
    if (check_grid(g, &d) != VERIS_OK || (elem_size != 4 && elem_size != 8) || n_subcycles < 0) return 0;
    return residual_workspace_bytes(d, (size_t)elem_size, n_subcycles);
}

int veris_evp_residual_solver_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs,
                                  int32_t n, double *u, double *v, double *s1, double *s2, double *s12,
                                  double *resU, double *resSig, void *ws, size_t ws_bytes, veris_stream_t s) {
    return evp_residual_solver<double>(g, p, reinterpret_cast<const Fields<double> *>(vs), n, u, v, s1, s2, s12,
                                       resU, resSig, ws, ws_bytes, s);
}

int veris_evp_residual_solver_f32(const VerisGrid *g, const VerisParams *p, const VerisFieldsF32 *vs,
                                  int32_t n, float *u, float *v, float *s1, float *s2, float *s12,
                                  double *resU, double *resSig, void *ws, size_t ws_bytes, veris_stream_t s) {
    return evp_residual_solver<float>(g, p, reinterpret_cast<const Fields<float> *>(vs), n, u, v, s1, s2, s12,
                                      resU, resSig, ws, ws_bytes, s);
}

size_t veris_evp_workspace_bytes(const VerisGrid *g, int32_t elem_size) {
    Dims d;
    if (check_grid(g, &d) != VERIS_OK || (elem_size != 4 && elem_size != 8)) return 0;
    return 5 * round_up(field_bytes(d, (size_t)elem_size), 256);
}

int veris_evp_solver_f64(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs, int32_t n,
                         double *u, double *v, double *s1, double *s2, double *s12, void *ws,
                         size_t ws_bytes, veris_stream_t s) {
    return evp_solver<double>(g, p, reinterpret_cast<const Fields<double> *>(vs), n, u, v, s1, s2, s12, ws,
                              ws_bytes, s);
}

int veris_evp_solver_f32(const VerisGrid *g, const VerisParams *p, const VerisFieldsF32 *vs, int32_t n,
                         float *u, float *v, float *s1, float *s2, float *s12, void *ws, size_t ws_bytes,
                         veris_stream_t s) {
    return evp_solver<float>(g, p, reinterpret_cast<const Fields<float> *>(vs), n, u, v, s1, s2, s12, ws,
                             ws_bytes, s);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free form of veris_evp_solver_f64 (no counterpart in the
// reference).  Some callers cannot allocate device memory: a host ocean
// model's time loop that drives the sea-ice step through this C ABI has no
// device allocator of its own, and a caller running under a device-memory
// budget fixed at start-up must not grow it per step.  For them the
// ping-pong half of the subcycle loop lives in this file-scope array instead
// of a caller-provided workspace.  Every GPU that loads the library holds the
// array until the process exits.  Nothing in it has to start at zero: each
// subcycle writes every point of the buffer before the next one reads it.
// Calls share the array, so calls that overlap on the GPU race on it.
namespace {

constexpr int64_t NOALLOC_MAX_CELLS = VERIS_NOALLOC_MAX_CELLS;
static __device__ __align__(256) double g_noalloc_scratch[5 * NOALLOC_MAX_CELLS];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
double *g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};

// device address of the scratch for the current device, looked up once per
// device with that device current
int noalloc_scratch(double **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return VERIS_ERR_LAUNCH;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) {
            cudaGetLastError();
            return VERIS_ERR_LAUNCH;
        }
        g_noalloc_ptr[dev] = static_cast<double *>(ptr);
    }
    *out = g_noalloc_ptr[dev];
    return VERIS_OK;
}

}  // namespace

extern "C" int veris_evp_solver_f64_noalloc(const VerisGrid *g, const VerisParams *p, const VerisFieldsF64 *vs,
                                            int32_t n, double *u, double *v, double *s1, double *s2, double *s12,
                                            veris_stream_t s) {
    Dims d;
    VERIS_CHECK_GRID(g, d);
    if ((int64_t)d.NX * d.ld > NOALLOC_MAX_CELLS) return VERIS_ERR_TOO_LARGE;
    VERIS_REQUIRE(p && vs && u && v && s1 && s2 && s12, VERIS_ERR_ARG);
    VERIS_REQUIRE(n >= 0, VERIS_ERR_ARG);
    double *scratch = nullptr;
    const int st = noalloc_scratch(&scratch);
    if (st != VERIS_OK) return st;
    // the five scratch buffers follow each other at NX * ld elements
    const size_t per = (size_t)d.NX * d.ld;
    const size_t need = 5 * round_up(per * sizeof(double), 256);
    return evp_solver<double>(g, p, reinterpret_cast<const Fields<double> *>(vs), n, u, v, s1, s2, s12, scratch,
                              need <= sizeof(g_noalloc_scratch) ? need : 0, s);
}
