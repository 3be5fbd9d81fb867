// nd_tile.h -- the TMA-staged tile pass's launcher: its kernels depend on the precision, not on the
// state count, so they are compiled in a unit of their own (nd_tile.cu, once per precision).
#pragma once

#include "nd_kernels.cuh"

namespace zqd {

constexpr int ND_TMA_LOGN_MIN = 5; // lines of 32 points and more take the TMA-staged passes

// the largest line of a d-dimensional grid the TMA-staged passes are built for (log2 of its points)
template <typename T> constexpr int nd_tma_logn_max(int d) { return d == 3 ? 10 : sizeof(T) == 8 ? 11 : 12; }

// resident CTAs per SM of the tile kernel for lines of 2^logn points (sets its shared-memory limit)
int nd_tile_per_sm_d(int d, int logn, int threads, size_t smem, int* per_sm);
int nd_tile_per_sm_f(int d, int logn, int threads, size_t smem, int* per_sm);
int nd_tile_launch_d(int logn, const NdJob<double>& J, const CUtensorMap& map, const NdTma& P, size_t part_base, const NdFin& F,
                     unsigned grid, unsigned threads, size_t smem, cudaStream_t st);
int nd_tile_launch_f(int logn, const NdJob<float>& J, const CUtensorMap& map, const NdTma& P, size_t part_base, const NdFin& F,
                     unsigned grid, unsigned threads, size_t smem, cudaStream_t st);
template <typename T> int nd_tile_per_sm(int d, int logn, int threads, size_t smem, int* per_sm) {
    if constexpr (sizeof(T) == 8) return nd_tile_per_sm_d(d, logn, threads, smem, per_sm);
    else return nd_tile_per_sm_f(d, logn, threads, smem, per_sm);
}
template <typename T>
int nd_tile_launch(int logn, const NdJob<T>& J, const CUtensorMap& map, const NdTma& P, size_t part_base, const NdFin& F,
                   unsigned grid, unsigned threads, size_t smem, cudaStream_t st) {
    if constexpr (sizeof(T) == 8) return nd_tile_launch_d(logn, J, map, P, part_base, F, grid, threads, smem, st);
    else return nd_tile_launch_f(logn, J, map, P, part_base, F, grid, threads, smem, st);
}

} // namespace zqd
