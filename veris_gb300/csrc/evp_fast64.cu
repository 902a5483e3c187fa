// Float64 fast-form subcycle: dispatch over the unit height, the drag options
// and the tape (the kernel is in evp_fast64.cuh).
#include "evp_fast64.cuh"

namespace veris {

// a taped subcycle (io.tDel set) also writes Delta, zeta and cDrag
template <int TI, bool B, bool R>
static int launch64_tape(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c,
                         const F64Scalars &k, const FastIO<double> &io, cudaStream_t st) {
    return io.tDel ? launch64<TI, B, R, true>(d, lp, h, c, k, io, st) : launch64<TI, B, R, false>(d, lp, h, c, k, io, st);
}

template <int TI>
static int launch64_rows(const Dims &d, int64_t lp, const HaloFill &h, const FastConsts<double> &c,
                         const F64Scalars &k, const FastIO<double> &io, bool basal, bool turn, cudaStream_t st) {
    if (basal)
        return turn ? launch64_tape<TI, true, true>(d, lp, h, c, k, io, st)
                    : launch64_tape<TI, true, false>(d, lp, h, c, k, io, st);
    return turn ? launch64_tape<TI, false, true>(d, lp, h, c, k, io, st)
                : launch64_tape<TI, false, false>(d, lp, h, c, k, io, st);
}

// rows per tile of later float64 subcycles (0: the default); process-wide
static std::atomic<int> g_tile_rows{0};
// 24 rows 171.5 us per subcycle on 1440x720 (unchained, cold start), 16 rows
// 172.5, 32 rows 202.1; 3600x1800 927 us (24) and 933 (16); the bench's tuner
// picks per workload
constexpr int F64_DEFAULT_ROWS = 24;

int fast64_subcycle(const Dims &d, const HaloFill &h, const FastConsts<double> &c, const FastScalars<double> &ks,
                    const FastIO<double> &io, bool basal, bool turn, cudaStream_t st) {
    const int64_t lp = internal_pitch(d.NY);
    const F64Scalars k = f64_scalars(ks);
    const int rows = g_tile_rows.load(std::memory_order_relaxed);
    switch (rows ? rows : F64_DEFAULT_ROWS) {
        case 16: return launch64_rows<16>(d, lp, h, c, k, io, basal, turn, st);
        case 24: return launch64_rows<24>(d, lp, h, c, k, io, basal, turn, st);
        default: return launch64_rows<32>(d, lp, h, c, k, io, basal, turn, st);
    }
}

}  // namespace veris

using namespace veris;

extern "C" int veris_evp_f64_tile_rows(int32_t rows) {
    VERIS_REQUIRE(rows == 0 || rows == 16 || rows == 24 || rows == 32, VERIS_ERR_ARG);
    g_tile_rows.store(rows, std::memory_order_relaxed);
    return VERIS_OK;
}
