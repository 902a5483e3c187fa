// Residual diagnostics of the EVP loop: the sums after one subcycle (evp.cu).
#pragma once

#include "common.cuh"

namespace veris {

constexpr int RES_THREADS = 256, RES_MAX_BLOCKS = 2048;

// one block per interior row (rows beyond RES_MAX_BLOCKS go round again)
inline int res_blocks(const Dims &d) { return d.nx < RES_MAX_BLOCKS ? d.nx : RES_MAX_BLOCKS; }

template <class T>
struct ResIO {
    const T *u0, *v0, *s10, *s20, *s120;   // before the subcycle
    const T *u1, *v1, *s11, *s21, *s121;   // after it
    const T *mC, *mU, *mV;
    const T *aC;                            // adaptive alphaC, or null: alpha and beta are constants
    double alpha, beta;
};

// the partial sums of one subcycle into partial[2 * res_blocks(d)]
template <class T>
int residual_partial(const Dims &d, const ResIO<T> &r, double *partial, cudaStream_t st);
// the sums of n subcycles from their partials, in index order
int residual_finish(const Dims &d, const double *partial, int n, double *resU, double *resSig, cudaStream_t st);

}  // namespace veris
