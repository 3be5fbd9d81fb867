// line_inst.cu -- instantiations of the resident line kernel for one
// (precision, state count) pair.  The build compiles this file once per pair
// with -DZQD_T=<double|float> -DZQD_S=<1..4> -DZQD_LAUNCH=<symbol> -DZQD_SERVICE=<symbol>
// -DZQD_ROOM=<symbol>, so the heavy template instantiations spread over parallel nvcc processes.
#include <algorithm>
#include <mutex>

#include "internal.h"
#include "line_solve.cuh"

#if !defined(ZQD_T) || !defined(ZQD_S) || !defined(ZQD_LAUNCH) || !defined(ZQD_SERVICE) || !defined(ZQD_ROOM)
#error "line_inst.cu needs -DZQD_T, -DZQD_S, -DZQD_LAUNCH, -DZQD_SERVICE and -DZQD_ROOM"
#endif

namespace zqd {

// The largest dynamic shared memory (a multiple of `grain`, at least `smem` rounded up to one) that leaves
// as many CTAs of the kernel on an SM as `smem` does.
static int room_of(const void* kern, int threads, size_t smem, size_t grain, size_t* room) {
    int dev = 0, total = 0, reserved = 0, per_sm = 0;
    cudaFuncAttributes fa{};
    ZQD_CUDA(cudaGetDevice(&dev));
    ZQD_CUDA(cudaDeviceGetAttribute(&total, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    ZQD_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
    ZQD_CUDA(cudaFuncGetAttributes(&fa, kern));
    *room = smem = (smem + grain - 1) / grain * grain;
    ZQD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    if (per_sm < 1) return ZQD_OK;
    const size_t each = (size_t)(total / per_sm), own = (size_t)reserved + fa.sharedSizeBytes;
    if (each <= own) return ZQD_OK;
    for (size_t most = std::min<size_t>(each - own, 215 * 1024) / grain * grain; most > smem; most -= grain) {
        int n = 0;
        ZQD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, most));
        if (n >= per_sm) { // at once, or a step of the hardware's allocation unit further down
            *room = most;
            return ZQD_OK;
        }
    }
    return ZQD_OK;
}

// launches njobs jobs, or (room != null) the shared memory a launch of this shape may take (room_of)
template <int C, int LRM, int MAXT = LineMaxThreads<ZQD_T>::value>
static int launch_one(const LaunchShape* J, const void* d_jobs, int njobs, size_t* room = nullptr) {
    auto kern = line_solve_kernel<ZQD_T, ZQD_S, C, LRM, MAXT>;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [&] {
        attr_err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 215 * 1024);
        if (attr_err == cudaSuccess && C > 8)
            attr_err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    });
    ZQD_CUDA(attr_err);
    if (room) return room_of((const void*)kern, J->threads, J->smem, 1024, room);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * njobs, 1, 1);
    cfg.blockDim = dim3(J->threads, 1, 1);
    cfg.dynamicSmemBytes = J->smem;
    cfg.stream = J->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ZQD_CUDA(cudaLaunchKernelEx(&cfg, kern, reinterpret_cast<const LineJob<ZQD_T>*>(d_jobs)));
    return ZQD_OK;
}

// A radix-4 launch of C-CTA clusters: FP32 CTAs of at most 256 threads take the form compiled for
// 256 threads (up to 255 registers, no spills; the FP32 kernel is otherwise compiled for 512-thread
// CTAs and 128 registers)
template <int C> static int launch_r4(const LaunchShape* J, const void* dj, int nj, size_t* room) {
    if (LineMaxThreads<ZQD_T>::value > 256 && J->threads <= 256) return launch_one<C, 2, 256>(J, dj, nj, room);
#if ZQD_S == 3
    // three states on 512-point CTAs: 384 threads, 168 registers instead of 128
    if constexpr (LineMaxThreads<ZQD_T>::value > 256)
        if (J->threads <= 384) return launch_one<C, 2, 384>(J, dj, nj, room);
#endif
    return launch_one<C, 2>(J, dj, nj, room);
}

// Radix-4 kernels for every cluster size; radix 8 only with 16 CTAs, the one shape whose CTAs can
// hold more points than radix-4 threads allow (the longest lines)
static int launch_form(const LaunchShape* J, const void* dj, int nj, size_t* room) {
    if (J->lrmax == 3) {
        if (J->C == 16) return launch_one<16, 3>(J, dj, nj, room);
        return fail(ZQD_ERR_UNSUPPORTED, "RADIX-8 LINE PASSES ARE BUILT FOR CLUSTERS OF 16 ONLY");
    }
    switch (J->C) {
    case 1: return launch_r4<1>(J, dj, nj, room);
    case 2: return launch_r4<2>(J, dj, nj, room);
    case 4: return launch_r4<4>(J, dj, nj, room);
    case 8: return launch_r4<8>(J, dj, nj, room);
    case 16: return launch_r4<16>(J, dj, nj, room);
    default: return fail(ZQD_ERR_UNSUPPORTED, "CLUSTER SIZE MUST BE 1, 2, 4, 8 OR 16");
    }
}
int ZQD_LAUNCH(const LaunchShape* J, const void* dj, int nj) { return launch_form(J, dj, nj, nullptr); }

// The persistent service kernel (single-CTA jobs, radix-4 local passes): grid CTAs of `threads`
// threads with `smem` bytes of dynamic shared memory each, on stream st.
// (always the form compiled for LineMaxThreads: its many small CTAs share SMs, which fewer
// registers per thread allow)
static int service_ready() {
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [&] {
        attr_err = cudaFuncSetAttribute(line_service_kernel<ZQD_T, ZQD_S, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 215 * 1024);
    });
    ZQD_CUDA(attr_err);
    return ZQD_OK;
}
int ZQD_SERVICE(const void* svc, unsigned grid, int threads, size_t smem, cudaStream_t st) {
    auto kern = line_service_kernel<ZQD_T, ZQD_S, 2>;
    if (const int rc = service_ready()) return rc;
    kern<<<grid, threads, smem, st>>>(*reinterpret_cast<const LineService<ZQD_T>*>(svc));
    ZQD_CUDA(cudaGetLastError());
    return ZQD_OK;
}

// The dynamic shared memory that jobs of this shape (J->smem: what they cannot do without) may use with as
// many CTAs per SM as without the extra: room in the line kernel, svc in the service kernel where that could
// take them (one CTA, radix 4; its CTAs' threads are a power of two and their memory a multiple of
// 16 KiB), else the same.
int ZQD_ROOM(const LaunchShape* J, size_t* room, size_t* svc) {
    if (const int rc = launch_form(J, nullptr, 0, room)) return rc;
    *svc = *room;
    if (J->C != 1 || J->lrmax != 2) return ZQD_OK;
    int threads = 64;
    while (threads < J->threads) threads <<= 1;
    if (const int rc = service_ready()) return rc;
    return room_of((const void*)line_service_kernel<ZQD_T, ZQD_S, 2>, threads, J->smem, 16384, svc);
}

} // namespace zqd
