// Work units of a tiled subcycle launch: which rows and columns a CTA takes.
#pragma once

#include "common.cuh"

namespace veris {

constexpr int UNIT_COLS = 32;

// Work units, one per CTA, in dispatch order: first the P1 pieces of rows
// [0, R1) of every 32-column strip, then the P2 smaller pieces of rows
// [R1, NX) of every strip (at most TI rows each, for which the shared memory
// is sized).  The hardware hands CTAs to SMs in block order as slots free up,
// so the launch ends on the small pieces and the SMs run out of work
// together instead of on a thin last wave of full tiles.
struct TileUnits {
    int P1, R1, P2, U1, count;
    __device__ __forceinline__ void unit(int b, int NX, int &i0, int &ti, int &j0) const {
        const bool big = b < U1;
        const int P = big ? P1 : P2, v = big ? b : b - U1;
        const int r0 = big ? 0 : R1, rows = big ? R1 : NX - R1, pc = v % P;
        i0 = r0 + (int)((int64_t)pc * rows / P);
        ti = r0 + (int)((int64_t)(pc + 1) * rows / P) - i0;
        j0 = (v / P) * UNIT_COLS;
    }
};

// The units of a launch.  When full pieces of TI rows would fit the resident
// CTAs' slots at once, the rows are dealt out over all slots instead, down to
// two rows a piece: a subcycle of a small grid then takes the time of a short
// piece, although its ring is a larger part of the work (pieces of five rows
// do a third more than they store, of two rows twice as much).  Float64
// subcycles with 24-row pieces took 33-35 us on every grid up to 443 x 221
// (8 CTAs on 90 x 40, 96 on 360 x 180); over all slots 90 x 40 takes 9.5 us,
// 360 x 180 22.6, 443 x 221 30.7, 720 x 360 59.6 (69.8 before); one piece per
// SM 9.6, 26.6, 34.8, 69.8; one-row pieces 11.9 on 90 x 40, at least three
// rows 11.8 there.
// Larger grids get a last round of about one small piece (TI/4 rows) per slot
// at the bottom of every strip, the rest in full pieces.  (Equal full tiles
// left a thin last wave: 12 % of the SM cycles idle on 1440 x 720 with 24-row
// tiles; third-height last pieces took 197.2 us a launch there,
// quarter-height 193.0, fifth- and sixth-height 193.8.)
inline TileUnits tile_units(const Dims &d, int TI, int slots) {
    const int strips = (d.NY + UNIT_COLS - 1) / UNIT_COLS;
    TileUnits w;
    const int minP = (d.NX + TI - 1) / TI;
    w.P2 = 0;
    w.R1 = d.NX;
    if ((int64_t)strips * minP > slots) {
        const int small = TI / 4 > 4 ? TI / 4 : 4;
        w.P2 = (slots + strips - 1) / strips;
        const int r2 = w.P2 * small;
        if (r2 < d.NX / 2) w.R1 = d.NX - r2;
        else w.P2 = 0;
    }
    w.P1 = (w.R1 + TI - 1) / TI;
    if ((int64_t)strips * minP <= slots) {
        const int fit = slots / strips, two = d.NX / 2;
        const int pieces = fit < two ? fit : two;
        if (pieces > w.P1) w.P1 = pieces;
    }
    w.U1 = strips * w.P1;
    w.count = w.U1 + strips * w.P2;
    return w;
}

// CTAs of `kern` resident on the current device at once (0 when unavailable);
// per_sm: the call site's own record of the occupancy per device
template <class K>
inline int cta_slots(std::atomic<int> (&per_sm)[MAX_DEVICES], K kern, int threads, size_t smem) {
    const int dev = current_device();
    if (dev < 0) return 0;
    int per = per_sm[dev].load(std::memory_order_acquire);
    if (per == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess || per < 1) {
            cudaGetLastError();
            return 0;
        }
        per_sm[dev].store(per, std::memory_order_release);
    }
    return per * sm_count();
}

}  // namespace veris
