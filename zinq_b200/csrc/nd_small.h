// nd_small.h -- small 2-D grids: a range of whole time steps in one launch of one thread-block cluster.
//
// A step of the axis passes is two launches of 5-6 us each whatever the grid's size: a 32^2 step took
// as long as a 128^2 one.  Grids of up to 128^2 points have too little work for that, and fit one
// cluster: CTA c of the cluster owns the columns and the rows c n/C .. (c + 1) n/C, transforms its
// columns (forward FFT, kinetic phase, inverse FFT), then its rows (inverse FFT, R, observables, R,
// forward FFT), with a cluster barrier after each half.  The state goes between the halves through L2;
// what a CTA reads of the tables every step fits its L1 up to three states (128^2 x 4: R alone is 164 KB a CTA, read
// from L2).  The sums of a row wait in shared memory for a spare
// warp of CTA 0, which writes the observables row while the others transform the next step's columns.
// 128^2 x 2 states FP64: 13.1 -> 9.6 us a step, 64^2 x 1: 11.0 -> 7.3.
#pragma once

#include "nd_kernels.cuh"

namespace zqd {

constexpr int ND_SMALL_LOGN_MIN = 5, ND_SMALL_LOGN_MAX = 7;
// CTAs of the cluster: at least one warp of sixteen-point threads per state and CTA
inline int nd_small_ctas(int logn) { return logn == 5 ? 2 : logn == 6 ? 8 : 16; }

struct NdSmall {
    int i0, i1, iters; // rows of the solve recorded by this launch; row 0 is the initial state's
    uint32_t mask;     // the observables of a row (no momentum-space ones)
    int ldx;           // exchange line stride
    double* hist;      // row 0 of the solve
    int hc;            // doubles per row
    int* rows_out;     // rows recorded so far
};

// launches the kernel for (precision, S, n = 2^logn) on J's stream
int nd_small_launch_d(int S, int logn, const NdJob<double>& J, const NdSmall& P, cudaStream_t st);
int nd_small_launch_f(int S, int logn, const NdJob<float>& J, const NdSmall& P, cudaStream_t st);
template <typename T> int nd_small_launch(int S, int logn, const NdJob<T>& J, const NdSmall& P, cudaStream_t st) {
    if constexpr (sizeof(T) == 8) return nd_small_launch_d(S, logn, J, P, st);
    else return nd_small_launch_f(S, logn, J, P, st);
}

} // namespace zqd
