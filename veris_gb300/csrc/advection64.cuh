// The float64 advection in two launches (advection64.cu).
#pragma once

#include "stencil.cuh"

namespace veris {

struct Adv64IO {
    const double *field[3];   // before advection
    double *f1[3];            // after the zonal update
    double *out[3];           // after the meridional update, masked; may be field
};

// settings and grids that it covers
bool advect64_covers(const VerisParams &p, const Dims &d);
// one field or three
int advect64(const Ctx<double> &c, const HaloFill &h, const Adv64IO &io, int nf, cudaStream_t st);

}  // namespace veris
