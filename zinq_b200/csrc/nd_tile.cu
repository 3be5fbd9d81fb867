// nd_tile.cu -- instantiations of the TMA-staged tile pass for one precision.  Compiled once per
// precision with -DZQD_T=<double|float> -DZQD_ND_TILE_PER_SM=<symbol> -DZQD_ND_TILE_LAUNCH=<symbol>.
#include "internal.h"
#include "nd_tile.h"

#if !defined(ZQD_T) || !defined(ZQD_ND_TILE_PER_SM) || !defined(ZQD_ND_TILE_LAUNCH)
#error "nd_tile.cu needs -DZQD_T, -DZQD_ND_TILE_PER_SM and -DZQD_ND_TILE_LAUNCH"
#endif

namespace zqd {
namespace {

using T = ZQD_T;
using Kernel = void (*)(NdJob<T>, CUtensorMap, NdTma, size_t, NdFin);

template <int D, int LOGN> Kernel pick(int logn, bool scale) {
    if constexpr (LOGN > nd_tma_logn_max<T>(D)) return nullptr;
    else if (logn != LOGN) return pick<D, LOGN + 1>(logn, scale);
    else return scale ? nd_tile_tma_kernel<T, D, LOGN, true> : nd_tile_tma_kernel<T, D, LOGN, false>;
}
Kernel tile_kernel(int d, int logn, bool scale) {
    return d == 2 ? pick<2, ND_TMA_LOGN_MIN>(logn, scale) : pick<3, ND_TMA_LOGN_MIN>(logn, scale);
}

} // namespace

int ZQD_ND_TILE_PER_SM(int d, int logn, int threads, size_t smem, int* per_sm) {
    const Kernel k = tile_kernel(d, logn, false), scaling = tile_kernel(d, logn, true);
    if (!k) return fail(ZQD_ERR_UNSUPPORTED, "LINE LENGTH OUTSIDE THE TMA-STAGED TILE PASS");
    ZQD_CUDA(cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, ND_SMEM_BUDGET));
    ZQD_CUDA(cudaFuncSetAttribute((const void*)scaling, cudaFuncAttributeMaxDynamicSharedMemorySize, ND_SMEM_BUDGET));
    ZQD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, (const void*)k, threads, smem));
    return ZQD_OK;
}

int ZQD_ND_TILE_LAUNCH(int logn, const NdJob<T>& J, const CUtensorMap& map, const NdTma& P, size_t part_base, const NdFin& F,
                       unsigned grid, unsigned threads, size_t smem, cudaStream_t st) {
    const Kernel k = tile_kernel(J.d, logn, P.mode & TM_SCALE);
    if (!k) return fail(ZQD_ERR_UNSUPPORTED, "LINE LENGTH OUTSIDE THE TMA-STAGED TILE PASS");
    k<<<grid, threads, smem, st>>>(J, map, P, part_base, F);
    ZQD_CUDA(cudaGetLastError());
    return ZQD_OK;
}

} // namespace zqd
