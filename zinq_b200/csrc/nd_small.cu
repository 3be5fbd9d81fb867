// nd_small.cu -- the one-cluster kernel for small 2-D grids (nd_small.h), compiled once per precision
// with -DZQD_T=<double|float> -DZQD_ND_SMALL_LAUNCH=<symbol>.
#include <cooperative_groups.h>

#include "internal.h"
#include "nd_small.h"

#if !defined(ZQD_T) || !defined(ZQD_ND_SMALL_LAUNCH)
#error "nd_small.cu needs -DZQD_T and -DZQD_ND_SMALL_LAUNCH"
#endif

namespace zqd {
namespace {
namespace cg = cooperative_groups;

using T = ZQD_T;

// The CTA's sums over its nt working threads, compensated, into out[v] = (sum, compensation) of each value
// set in act.  red: eight doubles a thread.  Called by the working threads only.
template <int NV>
__device__ __forceinline__ void worker_sums(const double (&a)[NV], uint32_t act, double* __restrict__ red,
                                            double (*__restrict__ out)[2], int nt, const SyncBar& all) {
    const int tid = threadIdx.x, lane = tid & 31, nw = nt >> 5, nact = __popc(act);
    for (int c0 = 0; c0 < nact; c0 += 8) {
        all();
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int k = __popc(act & ((1u << v) - 1u)) - c0;
            if (((act >> v) & 1u) && k >= 0 && k < 8) red[k * nt + tid] = a[v];
        }
        all();
        for (int k = tid >> 5; k < 8 && c0 + k < nact; k += nw) {
            Acc t;
            for (int e = lane; e < nt; e += 32) t.add(red[k * nt + e]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const double s2 = __shfl_down_sync(0xffffffffu, t.s, off), c2 = __shfl_down_sync(0xffffffffu, t.c, off);
                t.add(s2);
                t.c += c2;
            }
            if (lane == 0) {
                const int v = __fns(act, 0, c0 + k + 1);
                out[v][0] = t.s;
                out[v][1] = t.c;
            }
        }
    }
}

// 32 spare threads (the row writer) beside S n/C n/16 working ones
template <int S, int LOGN>
__global__ void __launch_bounds__(S * 64 + 32, 1)
    nd_small_kernel(const __grid_constant__ NdJob<T> J, const __grid_constant__ NdSmall P) {
    using PL = LinePlan<LOGN>;
    using SL = Slots<2, S>;
    constexpr int n = PL::n, TPL = PL::TPL;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double sums[2][SL::count][2]; // of the row in hand and the one before
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), cta = (int)cl.block_rank();
    const int L = n / C, nt = S * L * TPL, tid = threadIdx.x, lines = S * L; // L rows, L columns per CTA
    cx<T>* exch = reinterpret_cast<cx<T>*>(smem_raw);
    Tab<T>* tw = reinterpret_cast<Tab<T>*>(smem_raw + (((size_t)lines * P.ldx * sizeof(cx<T>) + 127) & ~(size_t)127));
    for (int t = tid; t < PL::ntw; t += blockDim.x) tw[t] = J.twd[t];
    __syncthreads();
    const SyncBar all{1, nt}; // the working threads
    const bool worker = tid < nt;
    uint32_t act = 1u << SL::norm;
    if (P.mask & WM_POS) act |= 3u << SL::pos;
    if (P.mask & WM_EPOT) act |= 1u << SL::epot;
    if (P.mask & WM_ACF) act |= 3u << SL::acf;
    if (P.mask & WM_POP) act |= ((1u << S) - 1u) << SL::pop;
    // the columns' threads sit side by side across columns (neighbouring threads, neighbouring addresses),
    // the rows' along the row; either way a line belongs to one warp
    constexpr int LPW = 32 / TPL;
    const int tg = (tid >> 5) * LPW + (tid & (LPW - 1)), ti = (tid & 31) / LPW; // column line s L + column, place
    const int rg = tid / TPL, ri = tid & (TPL - 1);                            // row line s L + row, place
    const SyncWarp sync{};
    // Row i of the solve: its sums (every CTA's, through distributed shared memory) to the history.
    auto write_row = [&](int i, int par) {
        const int v = tid & 31;
        Acc t;
        const bool have = v < SL::count && ((act >> v) & 1u);
        if (have)
            for (int c = 0; c < C; ++c) {
                const double* p = cl.map_shared_rank(&sums[par][v][0], c);
                t.add(p[0]);
                t.c += p[1];
            }
        double* row = P.hist + (size_t)i * P.hc;
        constexpr RowLayout R{2, S};
        const double x = t.value() * J.dr, nanv = nan("");
        if (v == SL::norm) row[R.norm()] = (P.mask & WM_NORM) ? x : nanv;
        if (v >= SL::pos && v < SL::pos + 2) row[R.pos() + v - SL::pos] = have ? x : nanv;
        if (v == SL::epot) row[R.epot()] = have ? x : nanv;
        if (v >= SL::acf && v < SL::acf + 2) row[R.acf() + v - SL::acf] = have ? x : nanv;
        if (v >= SL::mom && v < SL::mom + 2) row[R.mom() + v - SL::mom] = nanv;
        if (v == SL::ekin) row[R.ekin()] = nanv;
        if (v >= SL::pop && v < SL::pop + S) row[R.pop() + v - SL::pop] = have ? x : nanv;
        if (v == 0) *P.rows_out = i + 1;
    };
    for (int i = P.i0; i <= P.i1; ++i) {
        if (i > 0) {
            if (worker) { // columns: forward FFT, kinetic phase, inverse FFT
                const int s = tg / L, col = cta * L + (tg - s * L);
                cx<T>* g = J.psi + (size_t)s * J.N + col + (size_t)ti * n;
                cx<T>* line = exch + (size_t)tg * P.ldx;
                cx<T> v[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) v[t] = __ldcg(g + (size_t)t * TPL * n);
                line_fft<T, LOGN, -1>(v, line, ti, tw, sync);
                // exp(Complex(0, -K) * dt) as the product of per-axis factors (quantum_dynamics.zig:397-399)
                const double2 fl = J.kphase[n + col];
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    const double2 f = mul<double>(J.kphase[ti + t * TPL], fl);
                    v[t] = tmul<-1>(v[t], mktab<T>(f.x, f.y));
                }
                sync();
                line_fft<T, LOGN, 1>(v, line, ti, tw, sync);
#pragma unroll
                for (int t = 0; t < 16; ++t) __stcg(g + (size_t)t * TPL * n, v[t]);
            } else if (cta == 0 && i > P.i0) {
                write_row(i - 1, (i - 1) & 1); // beside the columns' work
            }
            cl.sync();
        }
        if (worker) { // rows: end of step i, its observables, start of step i + 1
            uint32_t mode = RM_OBS;
            if (i > 0) mode |= RM_INV | RM_REND;
            if (i < P.iters) mode |= RM_RSTART | RM_FWD;
            const int s = rg / L;
            const size_t row0 = (size_t)cta * L * n;
            cx<T>* g = J.psi + (size_t)s * J.N + row0 + (size_t)(rg - s * L) * n + ri;
            cx<T>* line = exch + (size_t)rg * P.ldx;
            cx<T> v[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = __ldcg(g + t * TPL);
            double acc[SL::count];
#pragma unroll
            for (int q = 0; q < SL::count; ++q) acc[q] = 0.0;
            all(); // the columns' lines of the exchange buffer belong to other threads
            if (mode & RM_INV) line_fft<T, LOGN, 1>(v, line, ri, tw, sync);
            if constexpr (S == 1) {
                nd_row_points<T, 2, true, SL::count, TPL>(J, v, row0 + (size_t)rg * n + ri, mode, P.mask, acc, (cx<T>*)nullptr,
                                                          [](int t) { return PL::pad_step(t); });
                sync();
            } else {
                sync();
                cx<T>* d = line + PL::pad(ri);
#pragma unroll
                for (int t = 0; t < 16; ++t) d[PL::pad_step(t)] = v[t];
                all();
                nd_row_sweep<T, 2, S, true, true, SL::count>(
                    J, exch, (cx<T>*)nullptr, [ldx = P.ldx](int ln, int x) { return ln * ldx + PL::pad(x); }, L, row0, mode, P.mask,
                    acc, nt, all);
#pragma unroll
                for (int t = 0; t < 16; ++t) v[t] = d[PL::pad_step(t)];
                sync();
            }
            if (mode & RM_FWD) line_fft<T, LOGN, -1>(v, line, ri, tw, sync);
#pragma unroll
            for (int t = 0; t < 16; ++t) __stcg(g + t * TPL, v[t]);
            worker_sums<SL::count>(acc, act, reinterpret_cast<double*>(exch), sums[i & 1], nt, all);
        }
        cl.sync(); // the rows and the sums are visible to the cluster
    }
    if (!worker && cta == 0) write_row(P.i1, P.i1 & 1);
    cl.sync(); // the sums stay until they have been read
}

template <int S, int LOGN> int launch(const NdJob<T>& J, const NdSmall& P, cudaStream_t st) {
    const int C = nd_small_ctas(LOGN), L = J.n / C, nt = S * L * J.n / 16;
    const size_t smem = (((size_t)S * L * P.ldx * sizeof(cx<T>) + 127) & ~(size_t)127) + (size_t)J.n * sizeof(Tab<T>);
    auto kern = nd_small_kernel<S, LOGN>;
    ZQD_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (C > 8) ZQD_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C, 1, 1);
    cfg.blockDim = dim3(nt + 32, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ZQD_CUDA(cudaLaunchKernelEx(&cfg, kern, J, P));
    return ZQD_OK;
}
template <int S> int launch_s(int logn, const NdJob<T>& J, const NdSmall& P, cudaStream_t st) {
    return logn == 5 ? launch<S, 5>(J, P, st) : logn == 6 ? launch<S, 6>(J, P, st) : launch<S, 7>(J, P, st);
}

} // namespace

int ZQD_ND_SMALL_LAUNCH(int S, int logn, const NdJob<T>& J, const NdSmall& P, cudaStream_t st) {
    if (logn < ND_SMALL_LOGN_MIN || logn > ND_SMALL_LOGN_MAX || J.d != 2) return fail(ZQD_ERR_UNSUPPORTED, "GRID OUTSIDE THE ONE-CLUSTER KERNEL");
    switch (S) {
    case 1: return launch_s<1>(logn, J, P, st);
    case 2: return launch_s<2>(logn, J, P, st);
    case 3: return launch_s<3>(logn, J, P, st);
    default: return launch_s<4>(logn, J, P, st);
    }
}

} // namespace zqd
