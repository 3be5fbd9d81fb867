// nd_inst.cu -- the 2-D / 3-D driver for one (precision, state count) pair.
// Compiled once per pair with -DZQD_T=<double|float> -DZQD_S=<1..4>
// -DZQD_ND_CREATE=<symbol> -DZQD_ND_RUN=<symbol> -DZQD_ND_STEP=<symbol>.
//
// A solve (src/quantum_dynamics.zig:860-950) is a stream-ordered sequence of
// axis passes (nd_kernels.cuh); nothing returns to the host until the end.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <utility>
#include <vector>

#include "job.h"
#include "nd_kernels.cuh"
#include "nd_small.h"
#include "nd_tile.h"

#if !defined(ZQD_T) || !defined(ZQD_S) || !defined(ZQD_ND_CREATE) || !defined(ZQD_ND_RUN) || !defined(ZQD_ND_STEP)
#error "nd_inst.cu needs -DZQD_T, -DZQD_S, -DZQD_ND_CREATE, -DZQD_ND_RUN and -DZQD_ND_STEP"
#endif

namespace zqd {
namespace {

using T = ZQD_T;
constexpr int S = ZQD_S;
constexpr int NSYM = S * (S + 1) / 2;

NdJob<T> describe(zqd_job* J) {
    NdJob<T> D{};
    const Opts& o = J->o;
    D.d = J->d;
    D.n = J->n;
    while ((1 << D.logn) < J->n) ++D.logn;
    D.S = S;
    D.N = J->N;
    for (int j = 0; j < D.d; ++j) {
        D.lo[j] = o.bounds[2 * j];
        D.span[j] = o.bounds[2 * j + 1] - o.bounds[2 * j];
        D.mass[j] = o.mass[j];
        D.dkunit[j] = 6.283185307179586476925286766559 / D.span[j];
        D.x0[j] = o.pos[j];
        D.p0[j] = o.mom[j];
        D.gamma[j] = o.gamma[j];
        if (o.has_cap) {
            D.cap_lo[j] = o.cap_bounds[2 * j];
            D.cap_hi[j] = o.cap_bounds[2 * j + 1];
        }
    }
    double dr = 1; // Grid.init (wavepacket.zig:44-53)
    for (int j = 0; j < D.d; ++j) dr *= D.span[j] / (double)J->n;
    D.dr = dr;
    D.dk = dr / (double)J->N;
    D.dt_re = o.imag_nstate ? 0.0 : o.time_step;
    D.dt_im = o.imag_nstate ? -o.time_step : 0.0;
    D.adiabatic = o.adiabatic;
    D.track = o.has_cap && o.cap_track;
    D.has_cap = o.has_cap;
    D.cap_exp = o.cap_exponent;
    D.ic_state = (int)o.ic_state;
    D.ic_adia = o.ic_adiabatic;
    D.psi = J->psi_save.as<cx<T>>();
    D.phi = J->phi.as<cx<T>>();
    D.psi0 = J->psi0.as<cx<T>>();
    D.psi_init = J->psi_init.as<cx<T>>();
    D.orth = J->orth.as<cx<T>>();
    D.R = J->R.as<Tab<T>>();
    D.V = J->V.as<double>();
    D.U = J->U.as<double>();
    D.capw = J->capw.as<double>();
    D.tw = J->tw.as<Tab<T>>();
    D.twd = D.tw + J->n;
    D.kphase = J->expk.as<double2>();
    D.axis = reinterpret_cast<const double4*>(J->expk.as<double2>() + (size_t)J->d * J->n);
    D.part = J->part.as<double>();
    D.nparts = J->part.bytes / (NDV * 2 * sizeof(double));
    D.rows_per_cta = J->nd_rows;
    D.tile = J->nd_tile;
    while ((1 << D.logtile) < J->nd_tile) ++D.logtile;
    D.stopped = J->flags.as<int>();
    D.err = J->flags.as<int>() + 2;
    D.nsum = J->book.as<NdBook>()->scal; // where nd_reduce_kernel leaves the norm's sum (device address)
    D.pot = J->pot.dev;
    return D;
}

// Row CTAs of at most 256 threads with several states take the 256-thread kernel form (up
// to 255 registers).  One state keeps the 512-thread form: its sweep fits in 128 registers
// and two 256-thread CTAs per SM hide more latency than extra registers would.
inline bool row_narrow(unsigned threads) { return S > 1 && threads <= 256; }

using RowTmaKernel = void (*)(NdJob<T>, NdRowTma, size_t);
// the longest line of the TMA-staged row pass: sixteen points a thread, at most 256 threads for the
// states of one row, and no longer than the tile pass's
constexpr int ROW_LOGN_MAX = S == 1 ? 12 : S == 2 ? 11 : 10;
template <int D, int LOGN> RowTmaKernel row_tma_pick(int logn, int form) {
    if constexpr (LOGN > ROW_LOGN_MAX || LOGN > nd_tma_logn_max<T>(D)) {
        return nullptr;
    } else {
        static const RowTmaKernel forms[RF_COUNT] = {
            nd_row_tma_kernel<T, D, S, LOGN, RF_GENERAL>, nd_row_tma_kernel<T, D, S, LOGN, RF_POP>,
            nd_row_tma_kernel<T, D, S, LOGN, RF_ACF>, nd_row_tma_kernel<T, D, S, LOGN, RF_ALL>};
        return logn == LOGN ? forms[form] : row_tma_pick<D, LOGN + 1>(logn, form);
    }
}
inline RowTmaKernel row_tma(int d, int logn, int form) {
    return d == 2 ? row_tma_pick<2, ND_TMA_LOGN_MIN>(logn, form) : row_tma_pick<3, ND_TMA_LOGN_MIN>(logn, form);
}
inline int log2_of(int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}
// exchange line stride of the two passes (exch_stride): rows take consecutive threads; a tile's lines
// sit side by side, those of a warp (tile_warp_lines) or all
inline int row_ldx(int n) { return exch_stride<T>(log2_of(n), 0); }
inline int tile_ldx(int n, int W) { return exch_stride<T>(log2_of(n), tile_warp_lines<T>(log2_of(n)) ? 512 / n : W); }

struct Launch {
    zqd_job* J;
    NdJob<T> D;
    size_t nrow_blocks, ntile_blocks, ngrid;
    size_t row_cols, k_cols; // partial-sum columns of a row launch and of a momentum launch
    // partial-sum regions (in blocks)
    size_t R0, R1, R2, K, G;
    NdFin ahead{}; // sums waiting for the next kinetic tile launch's extra CTA (FIN_AHEAD), if enabled

    // the waiting sums now, in a launch of their own
    int flush(bool nostop = false) {
        if (!ahead.enabled) return ZQD_OK;
        NdJob<T> d = D;
        if (nostop) d.stopped = J->flags.as<int>() + 1; // a flag nothing sets
        nd_finalize_kernel<T><<<1, 256, 0, J->stream>>>(d, ahead);
        ahead.enabled = 0;
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }

    // a row launch and, with momentum observables (RM_PHI), the launches that sum them, then the sums' reduction f:
    // by the last CTA of a per-block launch, at once (now), or by the next kinetic tile launch.
    int observe(uint32_t mode, uint32_t obs, size_t region, NdFin f, bool now, bool nostop = false, cx<T>* wout = nullptr) {
        // (per-block launches on large grids: 64^3 26.8 us a step against 28.3 with nd_finalize_kernel, where 32^3, 16^3
        // and 128^2 take 26.3, 24.6 and 21.1 with that against 27.3, 31.2 and 23.0)
        const bool k = mode & RM_PHI, own = (k ? !J->nd_tma : !J->nd_row_tma) && J->N >= ((size_t)1 << 18);
        int rc;
        f.enabled = own ? FIN_LAST : FIN_AHEAD;
        if ((rc = row(mode, obs, region, nostop, own && !k ? f : NdFin{}, wout))) return rc;
        if (k && (rc = kobs(nostop, own ? f : NdFin{}))) return rc;
        if (own) return ZQD_OK;
        ahead = f;
        return now ? flush(nostop) : ZQD_OK;
    }

    int row(uint32_t mode, uint32_t obs, size_t region, bool nostop = false, NdFin f = NdFin{}, cx<T>* wout = nullptr) {
        NdJob<T> d = D;
        d.wfn_out = wout;
        if (nostop) d.stopped = J->flags.as<int>() + 1; // a flag nothing sets
        if (J->nd_row_tma) {
            const bool phi = mode & RM_PHI;
            NdRowTma P{};
            P.mode = mode;
            P.obs = obs;
            P.logL = J->nd_row_tma_logL;
            P.nitems = (unsigned)(J->N / J->n >> P.logL);
            int form = RF_ALL;
            if (!(obs & ~row_form_obs(RF_POP))) form = RF_POP;
            else if (!(obs & ~row_form_obs(RF_ACF))) form = RF_ACF;
            if (d.track || d.wfn_out || (mode & RM_NORM)) form = RF_GENERAL;
            P.workers = (unsigned)(phi ? J->nd_row_phi_ctas : J->nd_row_ctas[form]);
            P.ncols = (unsigned)row_cols;
            P.shared = phi || J->nd_row_shared[form];
            P.ldx = row_ldx(J->n);
            bool withhold = false;
            P.wait_cycles = tma_wait_budget(NDT_WAIT_CYCLES, &withhold);
            P.withhold = withhold;
            const size_t smem = ndt_smem<T>(S << P.logL, J->n, P.ldx, P.shared, phi, row_ntw(form, J->n)).total;
            const unsigned nt = (unsigned)((S * J->n << P.logL) / 16);
            const RowTmaKernel kern = row_tma(D.d, D.logn, form);
            kern<<<P.workers, nt, smem, J->stream>>>(d, P, region);
            ZQD_CUDA(cudaGetLastError());
            return ZQD_OK;
        }
        const size_t smem = nd_smem_bytes<T>(2, S * J->nd_rows, J->n);
        const unsigned nb = (unsigned)nrow_blocks, nt = (unsigned)J->nd_row_threads;
        if (row_narrow(nt)) {
            if (D.d == 2) nd_row_kernel<T, 2, S, 256><<<nb, nt, smem, J->stream>>>(d, mode, obs, region, f);
            else nd_row_kernel<T, 3, S, 256><<<nb, nt, smem, J->stream>>>(d, mode, obs, region, f);
        } else {
            if (D.d == 2) nd_row_kernel<T, 2, S, 512><<<nb, nt, smem, J->stream>>>(d, mode, obs, region, f);
            else nd_row_kernel<T, 3, S, 512><<<nb, nt, smem, J->stream>>>(d, mode, obs, region, f);
        }
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    int tile(int axis, uint32_t mode, size_t region, bool nostop = false, NdFin f = NdFin{}) {
        NdJob<T> d = D;
        if (nostop) d.stopped = J->flags.as<int>() + 1;
        const size_t smem = nd_smem_bytes<T>(2, J->nd_tile, J->n);
        const dim3 grid((unsigned)ntile_blocks, S);
        if (D.d == 2) nd_tile_kernel<T, 2><<<grid, J->nd_tile_threads, smem, J->stream>>>(d, axis, mode, region, f);
        else nd_tile_kernel<T, 3><<<grid, J->nd_tile_threads, smem, J->stream>>>(d, axis, mode, region, f);
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    // the TMA-staged persistent form of a tile pass: over psi (modes TM_FWD, TM_KPHASE, TM_INV) or
    // over phi (TM_FWD, or TM_FWD | TM_KOBS: the momentum sums into region `region`)
    // (f: an earlier launch's sums, for an extra CTA)
    int tile_tma(int axis, uint32_t mode, bool phi = false, size_t region = 0, bool nostop = false, NdFin f = NdFin{}) {
        NdJob<T> d = D;
        if (nostop) d.stopped = J->flags.as<int>() + 1;
        const CUtensorMap* map = reinterpret_cast<const CUtensorMap*>(phi ? J->nd_maps_phi[axis] : J->nd_maps[axis]);
        NdTma P{};
        P.axis = axis;
        P.mode = mode;
        P.logW = J->nd_tma_logW;
        const int lstride = D.logn * (D.d - 1 - axis);
        int logN = 0;
        while (((size_t)1 << logN) < J->N) ++logN;
        P.logtiles = logN - D.logn - P.logW;
        P.logO = logN - D.logn - lstride;
        P.nitems = (unsigned)S << P.logtiles;
        P.shared = J->nd_tma_shared;
        P.ldx = tile_ldx(J->n, 1 << P.logW);
        const size_t smem = ndt_smem<T>(1 << P.logW, J->n, P.ldx, P.shared, false, J->n).total;
        const unsigned threads = (unsigned)((J->n << P.logW) / 16);
        P.workers = (unsigned)J->nd_tma_ctas;
        P.ncols = (unsigned)row_cols;
        if (phi) P.mode |= TM_PHI;
        bool withhold = false;
        P.wait_cycles = tma_wait_budget(NDT_WAIT_CYCLES, &withhold);
        P.withhold = withhold;
        return nd_tile_launch<T>(D.logn, d, *map, P, region, f, P.workers + (f.enabled == FIN_AHEAD), threads, smem, J->stream);
    }
    int ptile(int axis, uint32_t mode) {
        if (!J->nd_tma) {
            const int rc = flush();
            return rc ? rc : tile(axis, mode, 0);
        }
        // the waiting sums ride on the step's longest tile launch (128^3 FP32: the reduction takes 11 us, the
        // single-direction passes 8.5, the kinetic one 16)
        NdFin f{};
        if (mode & TM_KPHASE) std::swap(f, ahead);
        return tile_tma(axis, mode, false, 0, false, f);
    }
    // forward along axes d-2..1, forward + kinetic phase + inverse along axis 0, inverse along 1..d-2;
    // `first`: mode bits of the first of these launches only (TM_SCALE, whose sum is region R0's)
    int step_tiles(uint32_t first = 0) {
        int rc;
        for (int a = D.d - 2; a >= 1; --a, first = 0)
            if ((rc = ptile(a, TM_FWD | first))) return rc;
        if ((rc = ptile(0, TM_FWD | TM_KPHASE | TM_INV | first))) return rc;
        for (int a = 1; a <= D.d - 2; ++a)
            if ((rc = ptile(a, TM_INV))) return rc;
        return ZQD_OK;
    }
    double* scal() const { return J->book.as<NdBook>()->scal; }
    // Hamiltonian.update at time t (with_R: and Propagator.update); with sign tracking, the global
    // eigenvector alignment with the previous update follows (wavepacket.zig:157-167)
    int table(double t, int with_R) {
        if (!needs_sign_tracking(J->o, S, J->nsolve)) {
            nd_table_kernel<T, S><<<(unsigned)((J->N + 127) / 128), 128, 0, J->stream>>>(D, t, with_R);
            ZQD_CUDA(cudaGetLastError());
            return ZQD_OK;
        }
        const unsigned nb = (unsigned)std::min<size_t>(ngrid, (J->N + 127) / 128);
        nd_table_sign_kernel<T, S><<<nb, 128, 0, J->stream>>>(D, t, with_R, G);
        ZQD_CUDA(cudaGetLastError());
        int rc = reduce(G, G + nb, S);
        if (rc) return rc;
        nd_sign_flip_kernel<S><<<(unsigned)ngrid, 256, 0, J->stream>>>(D.U, J->N, scal(), D.stopped);
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    // scalar sums of slots [0, nv) over partial blocks [b0, b1) into scal()
    int reduce(size_t b0, size_t b1, int nv, bool clear = false) {
        nd_reduce_kernel<<<1, 32 * nv, 0, J->stream>>>(D.part, D.nparts, b0, b1, nv, D.stopped, scal(), clear ? 1 : 0);
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    // momentum observables of phi (the forward transform along the last axis is already done); f: the
    // per-block kernel's last CTA's reduction
    int kobs(bool nostop, NdFin f) {
        int rc;
        if (J->nd_tma) {
            for (int a = D.d - 2; a >= 1; --a)
                if ((rc = tile_tma(a, TM_FWD, true, 0, nostop))) return rc;
            return tile_tma(0, TM_FWD | TM_KOBS, true, K, nostop);
        }
        for (int a = D.d - 2; a >= 1; --a)
            if ((rc = tile(a, TM_FWD | TM_PHI, 0, nostop))) return rc;
        return tile(0, TM_FWD | TM_KOBS | TM_PHI, K, nostop, f);
    }
};

// Grid of a persistent pass: with room for every item at once the stage and the exchange buffer share
// their space (more CTAs fit); otherwise they are separate, so that a CTA's next load overlaps its work,
// where that still leaves two CTAs per SM.  per_sm(smem): resident CTAs per SM; extra: CTAs of the
// launch that take no items (they must not wait for a worker to leave).
template <typename F>
int choose_grid(size_t items, int sms, int extra, size_t smem_shared, size_t smem_apart, const F& per_sm, bool& shared,
                int& ctas) {
    int a = 0, b = 0, rc;
    if ((rc = per_sm(smem_shared, &a))) return rc;
    shared = true;
    if (items > (size_t)a * sms && smem_apart <= (size_t)ND_SMEM_BUDGET) {
        if ((rc = per_sm(smem_apart, &b))) return rc;
        if (b >= 2) shared = false;
    }
    ctas = (int)std::min<size_t>(items, (size_t)std::max(1, shared ? a : b) * sms - (size_t)extra);
    return ZQD_OK;
}

// A table's or the autotuner's shape for the TMA-staged passes names whole warps of eight points a thread, the
// threads these passes had when the first tables were measured, up to `most` of them; other shapes are
// refused.  (Sixteen points a thread: blocks that leave half a warp are widened.)
inline bool tuned_threads_ok(size_t points, size_t most) { return points / 8 % 32 == 0 && points / 8 <= most; }

// The TMA-staged tile pass: lines per tile W (a power of two, W <= n) with rows of W c >= 16
// bytes (an even number of 8-byte words), W n / 16 threads (whole warps, at most 256, 512 on lines of
// 4096 points) and the stage, exchange and
// twiddles within the shared-memory budget; by default the widest W up to 64-byte rows.  w_override
// (the autotuner's candidate or table entry): 0 keeps the default, -1 keeps the earlier tile
// kernel, else W.  ZQD_ND_TMA=0 in the environment also keeps it.
int setup_tma_shape(zqd_job* J, int w_override) {
    constexpr int c = (int)sizeof(cx<T>), E = c / 8;
    const int n = J->n, d = J->d, logn = log2_of(n);
    J->nd_tma = false;
    const char* env = getenv("ZQD_ND_TMA");
    if ((env && env[0] == '0') || w_override < 0) return ZQD_OK;
    if (w_override > 0 && (w_override > n || (E * w_override) % 2 || (J->N / n) % w_override || !tuned_threads_ok((size_t)w_override * n, 512)))
        return fail(ZQD_ERR_UNSUPPORTED, "TMA TILE SHAPE OUTSIDE THE KERNEL'S LIMITS");
    if (logn < ND_TMA_LOGN_MIN || logn > nd_tma_logn_max<T>(d)) return ZQD_OK; // the per-block kernels
    int dev = 0, sms = 148;
    ZQD_CUDA(cudaGetDevice(&dev));
    ZQD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t tmax = logn == 12 ? 512 : 256;
    auto fits = [&](int W) {
        const size_t t = (size_t)W * n / 16;
        return W >= 1 && W <= n && (E * W) % 2 == 0 && t <= tmax && t % 32 == 0 &&
               ndt_smem<T>(W, n, tile_ldx(n, W), true, false, n).total <= (size_t)ND_SMEM_BUDGET;
    };
    const size_t lines = J->N / (size_t)n; // lines of one state along any axis
    int W = 0;
    if (w_override > 0) W = w_override;
    if (W) {
        while (W < n && (size_t)W * n / 16 % 32) W <<= 1; // whole warps
        if (!fits(W) || lines % (size_t)W) return fail(ZQD_ERR_UNSUPPORTED, "TMA TILE SHAPE OUTSIDE THE KERNEL'S LIMITS");
    } else {
        // 64-byte rows, or 32-byte rows where that gives the device fewer than two tiles per SM (and the
        // lines of one warp where those are more)
        for (int w = std::max(64 / c, 512 / n); w >= 1 && !W; w >>= 1)
            if (fits(w) && lines % (size_t)w == 0 && (w * c <= 32 || (size_t)S * (lines / w) >= 2 * (size_t)sms || !fits(w / 2))) W = w;
        if (!W) return ZQD_OK; // no shape fits: the earlier tile kernel runs
    }
    const size_t items = (size_t)S * (lines / W);
    const int ldx = tile_ldx(n, W);
    int rc;
    if ((rc = choose_grid(items, sms, 1, ndt_smem<T>(W, n, ldx, true, false, n).total, ndt_smem<T>(W, n, ldx, false, false, n).total,
                          [&](size_t smem, int* per) { return nd_tile_per_sm<T>(d, logn, W * n / 16, smem, per); },
                          J->nd_tma_shared, J->nd_tma_ctas)))
        return rc;
    J->nd_tma_logW = log2_of(W);
    J->nd_tma = true;
    return ZQD_OK;
}

// the tile pass's tensor maps over psi and phi, one per strided axis (after they are allocated)
int encode_tile_maps(zqd_job* J) {
    constexpr int c = (int)sizeof(cx<T>), E = c / 8;
    const int n = J->n, d = J->d, logn = log2_of(n), W = 1 << J->nd_tma_logW;
    for (int a = 0; a + 1 < d; ++a) {
        const int lstride = logn * (d - 1 - a);
        const uint64_t st = (uint64_t)1 << lstride, O = J->N / ((uint64_t)n * st);
        const uint64_t dims[3] = {(uint64_t)E * st, (uint64_t)n, (uint64_t)S * O};
        const uint32_t box[3] = {(uint32_t)(E * W), (uint32_t)std::min(n, 256), 1};
        const int l2 = W * c >= 128 ? 128 : 0; // (promotion measured no faster on narrower rows)
        const int e = encode_map_3d(reinterpret_cast<CUtensorMap*>(J->nd_maps[a]), J->psi_save.p, dims, st * c,
                                    (uint64_t)n * st * c, box, l2) ||
                      encode_map_3d(reinterpret_cast<CUtensorMap*>(J->nd_maps_phi[a]), J->phi.p, dims, st * c,
                                    (uint64_t)n * st * c, box, l2);
        if (e) return fail(ZQD_ERR_DEVICE, "cuTensorMapEncodeTiled failed for the tile pass");
    }
    return ZQD_OK;
}

// The TMA-staged row pass: L rows (a power of two dividing N/n) per block, S L n / 16 threads (whole
// warps, at most 256) and the stage, exchange (and, for the momentum copy, its lines) and twiddles
// within the budget.  The grid takes every resident CTA (jobs created by the server too: its
// observables' sums are grouped per CTA, so a job's results depend on its grid, which must not change
// with where it runs).  l_override: 0 keeps the default, -1 keeps the earlier row kernel, else L.
// ZQD_ND_TMA=0 also keeps it.
int choose_row_tma(zqd_job* J, int l_override) {
    const int n = J->n, d = J->d, logn = log2_of(n), ldx = logn >= ND_TMA_LOGN_MIN ? row_ldx(n) : n;
    const size_t lines = J->N / (size_t)n;
    J->nd_row_tma = false;
    const char* env = getenv("ZQD_ND_TMA");
    if ((env && env[0] == '0') || l_override < 0) return ZQD_OK;
    if (l_override > 0 && ((size_t)l_override > lines || lines % (size_t)l_override || (size_t)l_override * n * sizeof(cx<T>) < 1024 ||
                           !tuned_threads_ok((size_t)S * l_override * n, S <= 2 ? 512 : 256)))
        return fail(ZQD_ERR_UNSUPPORTED, "TMA ROW-BLOCK SHAPE OUTSIDE THE KERNEL'S LIMITS");
    if (logn < ND_TMA_LOGN_MIN || !row_tma(d, logn, RF_GENERAL)) return ZQD_OK; // the per-block kernels
    int dev = 0, sms = 148;
    ZQD_CUDA(cudaGetDevice(&dev));
    ZQD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (int form = 0; form < RF_COUNT; ++form)
        ZQD_CUDA(cudaFuncSetAttribute((const void*)row_tma(d, logn, form), cudaFuncAttributeMaxDynamicSharedMemorySize, ND_SMEM_BUDGET));
    auto threads_of = [&](int L) { return (size_t)S * L * n / 16; };
    auto fits = [&](int L) {
        const size_t t = threads_of(L);
        return L >= 1 && (size_t)L <= lines && lines % (size_t)L == 0 && t % 32 == 0 && t <= (size_t)NDR_THREADS &&
               ndt_smem<T>(S * L, n, ldx, true, true, n).total <= (size_t)ND_SMEM_BUDGET;
    };
    int L = 0;
    if (l_override > 0) L = l_override;
    if (L) {
        while ((size_t)L < lines && threads_of(L) % 32) L <<= 1; // whole warps
        if (!fits(L)) return fail(ZQD_ERR_UNSUPPORTED, "TMA ROW-BLOCK SHAPE OUTSIDE THE KERNEL'S LIMITS");
    } else { // the smallest block of at least 64 threads; one FP32 state 128 while the device has a block per SM
        // (1024^2 28.3 -> 24.5 us a step, 128^3 49.0 -> 47.0; FP64 and several states lose: 128^3 x 2 FP64 134 -> 139)
        for (int l = 1; (size_t)l <= lines && !L; l <<= 1)
            if (fits(l) && (threads_of(l) >= 64 || !fits(2 * l))) L = l;
        if (!L) return ZQD_OK; // no shape fits: the earlier row kernel runs
        if (S == 1 && sizeof(T) == 4 && fits(2 * L) && threads_of(2 * L) <= 128 && lines / (2 * L) >= (size_t)sms) L <<= 1;
    }
    // each form's grid (their registers and twiddles differ), and the momentum copy's, which always shares
    auto smem_of = [&](int form, bool shared, bool copy) { return ndt_smem<T>(S * L, n, ldx, shared, copy, row_ntw(form, n)).total; };
    for (int form = 0; form <= RF_COUNT; ++form) {
        const bool copy = form == RF_COUNT;
        const int fk = copy ? (int)RF_ALL : form;
        auto per_sm = [&](size_t smem, int* per) -> int {
            ZQD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, (const void*)row_tma(d, logn, fk), (int)threads_of(L), smem));
            return ZQD_OK;
        };
        bool shared = true;
        int ctas = 0;
        if (const int rc = choose_grid(lines / L, sms, 0, smem_of(fk, true, copy),
                                       copy ? (size_t)ND_SMEM_BUDGET + 1 : smem_of(fk, false, false), per_sm, shared, ctas))
            return rc;
        if (copy) {
            J->nd_row_phi_ctas = ctas;
        } else {
            J->nd_row_ctas[form] = ctas;
            J->nd_row_shared[form] = shared;
        }
    }
    J->nd_row_tma_logL = log2_of(L);
    J->nd_row_tma = true;
    return ZQD_OK;
}

} // namespace

int ZQD_ND_CREATE(zqd_job* J) {
    const size_t N = J->N, c = sizeof(cx<T>), tb = sizeof(Tab<T>);
    const Opts& o = J->o;
    const int n = J->n;
    // Launch shapes.  Row pass: L rows (all S states) per CTA, about 2048 points a CTA, at
    // least two CTAs per SM where the grid allows, within the shared-memory budget (two line
    // buffers; one thread per 8-point group).
    // Tile pass: Tn lines per CTA, rows of Tn * c >= 32 bytes (one sector), shrunk from
    // 128 bytes until the grid has two CTAs per SM.
    const int budget = ND_SMEM_BUDGET, sms2 = 2 * 148;
    const int max_items = 512; // 8-point groups of a CTA, one thread each
    J->nd_row_bufs = 2;
    if (S * n > 8 * max_items) return fail(ZQD_ERR_UNSUPPORTED, "GRID LINE TOO LONG FOR THE ROW PASS (states x npoint at most 4096)");
    static_assert(ND_IPT == 1, "launch shapes assume one 8-point group per thread");
    int L = std::max(1, std::min<int>((int)(N / n), 2048 / (S * n)));
    while (L > 1 && (N / n / L < (size_t)sms2 || nd_smem_bytes<T>(J->nd_row_bufs, S * L, n) > (size_t)budget)) L >>= 1;
    if (nd_smem_bytes<T>(J->nd_row_bufs, S * L, n) > (size_t)budget)
        return fail(ZQD_ERR_UNSUPPORTED, "GRID LINE TOO LONG FOR THE ROW PASS");
    J->nd_rows = L;
    J->nd_row_threads = std::max(32, (S * L * n / 8 + 31) / 32 * 32);
    const int tmin = std::max(1, (int)(32 / c));
    int Tn = std::min(n, (int)(128 / c));
    // at most 256 threads, except that long lines keep one 32-byte sector per row (up to 512 threads)
    while (Tn > 1 && ((Tn * n / 8 > 256 && (Tn > tmin || Tn * n / 8 > max_items)) ||
                      nd_smem_bytes<T>(2, Tn, n) > (size_t)budget || (Tn > tmin && (size_t)S * (N / n / Tn) < (size_t)sms2)))
        Tn >>= 1;
    if (nd_smem_bytes<T>(2, Tn, n) > (size_t)budget || Tn * n / 8 > max_items)
        return fail(ZQD_ERR_UNSUPPORTED, "GRID LINE TOO LONG FOR THE TILE PASS");
    J->nd_tile = Tn;
    ShapeOverride ov; // autotuned shape (or a candidate the autotuner measures), within the same limits
    if (lookup_shape(J->d, n, S, J->fp32, ov)) {
        if (ov.rows) {
            if ((size_t)ov.rows > N / n || (N / n) % (size_t)ov.rows || S * ov.rows * n / 8 > max_items ||
                nd_smem_bytes<T>(J->nd_row_bufs, S * ov.rows, n) > (size_t)budget)
                return fail(ZQD_ERR_UNSUPPORTED, "ROW-PASS SHAPE OUTSIDE THE KERNEL'S LIMITS");
            J->nd_rows = L = ov.rows;
            J->nd_row_threads = std::max(32, (S * L * n / 8 + 31) / 32 * 32);
        }
        if (ov.tile) {
            if (ov.tile > n || (N / n) % (size_t)ov.tile || ov.tile * n / 8 > max_items ||
                nd_smem_bytes<T>(2, ov.tile, n) > (size_t)budget)
                return fail(ZQD_ERR_UNSUPPORTED, "TILE-PASS SHAPE OUTSIDE THE KERNEL'S LIMITS");
            J->nd_tile = Tn = ov.tile;
        }
    }
    J->nd_tile_threads = std::max(32, (Tn * n / 8 + 31) / 32 * 32);
    int rc;
    if ((rc = choose_row_tma(J, ov.tma_rows)) || (rc = setup_tma_shape(J, ov.tma_w))) return rc;
    // columns of the partial sums: one per CTA of a row launch or of a momentum launch
    J->nd_row_cols = (int)(N / n / L);
    if (J->nd_row_tma) J->nd_row_cols = std::max(J->nd_row_phi_ctas, *std::max_element(J->nd_row_ctas, J->nd_row_ctas + RF_COUNT));
    // a forced or tuned shape of the axis passes is theirs (a table's entry for such a grid, also one written before the
    // one-cluster kernel existed, keeps the axis passes; zqd_autotune writes one only where it beat that kernel)
    J->nd_small = J->d == 2 && J->nd_tma && J->nd_row_tma && log2_of(n) <= ND_SMALL_LOGN_MAX && !ov.rows && !ov.tile && !ov.tma_rows && !ov.tma_w;
    J->nd_k_cols = J->nd_tma ? J->nd_tma_ctas : (int)(S * (N / n / Tn));
    const size_t nparts = 3 * (size_t)J->nd_row_cols + J->nd_k_cols + 1024;
    if ((rc = J->psi_save.alloc((size_t)S * N * c, J->stream))) return rc;
    if ((rc = J->phi.alloc((size_t)S * N * c, J->stream))) return rc;
    if ((o.has_spectrum || (o.write_mask & ZQD_WRITE_ACF)) && (rc = J->psi0.alloc((size_t)S * N * c, J->stream))) return rc;
    if (o.imag_nstate > 1 && (rc = J->orth.alloc((size_t)(o.imag_nstate - 1) * S * N * c, J->stream))) return rc;
    if ((rc = J->R.alloc((size_t)NSYM * N * tb, J->stream))) return rc;
    if ((rc = J->V.alloc((size_t)S * S * N * sizeof(double), J->stream))) return rc;
    if (S > 1 && (rc = J->U.alloc((size_t)S * S * N * sizeof(double), J->stream))) return rc;
    if (o.has_cap && (rc = J->capw.alloc(N * sizeof(double), J->stream))) return rc;
    if ((rc = J->tw.alloc((size_t)2 * n * tb, J->stream))) return rc; // natural order, then pass by pass
    if ((rc = J->expk.alloc((size_t)J->d * n * (sizeof(double2) + sizeof(double4)), J->stream))) return rc; // phases, axis table
    if ((rc = J->part.alloc(nparts * NDV * 2 * sizeof(double), J->stream))) return rc;
    if ((o.write_mask & ZQD_WRITE_WAVEFUNCTION) &&
        (rc = J->wfn_hist.alloc((size_t)J->nsolve * (o.iterations + 1) * S * N * c, J->stream)))
        return rc;
    if (!o.ic_wfn.empty()) { // initial wavefunction, natural order
        if ((rc = J->psi_init.alloc((size_t)S * N * c, J->stream))) return rc;
        std::vector<cx<T>> h((size_t)S * N);
        for (size_t e = 0; e < (size_t)S * N; ++e) h[e] = mk<T>((T)o.ic_wfn[2 * e], (T)o.ic_wfn[2 * e + 1]);
        ZQD_CUDA(cudaMemcpyAsync(J->psi_init.p, h.data(), (size_t)S * N * c, cudaMemcpyHostToDevice, J->stream));
        ZQD_CUDA(cudaStreamSynchronize(J->stream));
        J->h2d += (size_t)S * N * c;
    }
    if ((rc = J->book.alloc(sizeof(NdBook), J->stream))) return rc;
    if ((rc = J->flags.alloc(4 * sizeof(int), J->stream))) return rc; // stopped, never set, TMA error, spare
    const size_t rows = (size_t)o.iterations + 1;
    if ((rc = J->hist.alloc((size_t)J->nsolve * rows * J->hc * sizeof(double), J->stream))) return rc;
    if ((rc = J->fin.alloc((size_t)J->nsolve * J->hc * sizeof(double), J->stream))) return rc;
    if ((rc = J->rows.alloc((size_t)J->nsolve * sizeof(int), J->stream))) return rc;
    J->device_bytes = J->psi_save.bytes + J->phi.bytes + J->psi0.bytes + J->orth.bytes + J->R.bytes + J->V.bytes +
                      J->U.bytes + J->capw.bytes + J->part.bytes + J->hist.bytes;
    std::vector<double> tw = twiddles_f64(n);
    std::vector<Tab<T>> twt(2 * (size_t)n);
    for (int t = 0; t < n; ++t) twt[t] = mktab<T>(tw[2 * t], tw[2 * t + 1]);
    dense_twiddles(log2_of(n), twt.data(), twt.data() + n);
    ZQD_CUDA(cudaMemcpyAsync(J->tw.p, twt.data(), 2 * (size_t)n * tb, cudaMemcpyHostToDevice, J->stream));
    ZQD_CUDA(cudaMemsetAsync(J->flags.p, 0, 4 * sizeof(int), J->stream));
    ZQD_CUDA(cudaMemsetAsync(J->hist.p, 0xff, J->hist.bytes, J->stream)); // NaN until written
    J->h2d += 2 * (size_t)n * tb + J->pot.bytes;
    NdJob<T> D = describe(J);
    nd_table_kernel<T, S><<<(unsigned)((N + 127) / 128), 128, 0, J->stream>>>(D, 0.0, 1);
    ZQD_CUDA(cudaGetLastError());
    nd_kphase_kernel<T><<<(unsigned)((J->d * n + 127) / 128), 128, 0, J->stream>>>(
        D, J->expk.as<double2>(), const_cast<double4*>(D.axis));
    ZQD_CUDA(cudaGetLastError());
    for (auto f : {nd_row_kernel<T, 2, S, 256>, nd_row_kernel<T, 3, S, 256>, nd_row_kernel<T, 2, S, 512>,
                   nd_row_kernel<T, 3, S, 512>})
        ZQD_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, budget));
    for (auto f : {nd_tile_kernel<T, 2>, nd_tile_kernel<T, 3>})
        ZQD_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, budget));
    if (J->nd_tma && (rc = encode_tile_maps(J))) return rc;
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    return ZQD_OK;
}

namespace {
// The launches of a run, in stream order, in three pieces per solve: the prologue (setGaussian,
// normalise, toDia), the launches of loop index i (step i, then the observables of row i) and the
// epilogue (final observables, orthw.append).  A whole run (enqueue) is every piece in order; a
// step range (ZQD_ND_STEP) is a run of consecutive loop indices.
struct Seq {
    zqd_job* J;
    Launch Lc;
    bool split, acf;
    int iters, HC;
    size_t SN;
    unsigned ng;

    explicit Seq(zqd_job* j) : J(j), Lc{j, describe(j)} {
        const Opts& o = J->o;
        const size_t N = J->N;
        Lc.nrow_blocks = N / J->n / J->nd_rows;
        Lc.ntile_blocks = N / J->n / J->nd_tile;
        Lc.ngrid = std::min<size_t>(1024, (N + 255) / 256);
        Lc.row_cols = (size_t)J->nd_row_cols;
        Lc.k_cols = (size_t)J->nd_k_cols;
        Lc.R0 = 0;
        Lc.R1 = Lc.row_cols;
        Lc.R2 = 2 * Lc.row_cols;
        Lc.K = 3 * Lc.row_cols;
        Lc.G = Lc.K + Lc.k_cols;
        split = o.imag_nstate > 0 || o.pot_td || (o.has_cap && o.cap_has_stop);
        acf = o.has_spectrum || (o.write_mask & ZQD_WRITE_ACF);
        iters = (int)o.iterations;
        HC = J->hc;
        SN = (size_t)S * N * sizeof(cx<T>);
        ng = (unsigned)Lc.ngrid;
        Lc.D.orth = J->orth.as<cx<T>>();
    }
    double* hist(int s) const { return J->hist.as<double>() + (size_t)s * (iters + 1) * HC; }
    int* rows_out(int s) const { return J->rows.as<int>() + s; }
    // Imaginary time, first state, no absorbing potential, no time-dependent potential and no
    // wavefunction history: the renormalisation of step i (quantum_dynamics.zig:898-906 with no
    // earlier states) is deferred.  Propagation is linear, the norm, populations, energies and
    // positions are quadratic in psi and the autocorrelation is linear, so the step closes and the
    // next one opens in a single row pass over the unnormalised psi, as in real time; its finalize
    // scales the observables row by the renormalisation factor (squared) and keeps the sum of
    // |psi|^2, and the first tile pass of step i+1 (or the final observables' pass) multiplies psi
    // by that factor as it loads it.
    bool deferred(int s) const {
        const Opts& o = J->o;
        return o.imag_nstate && s == 0 && !o.has_cap && !o.pot_td && !J->wfn_hist.p;
    }
    // Small 2-D grids in real time that record nothing in momentum space, track no absorption and keep no
    // wavefunction history run whole ranges of steps in one launch (nd_small.h).
    bool small() const {
        const Opts& o = J->o;
        return J->nd_small && !split && !o.log && !J->wfn_hist.p && !(o.has_cap && o.cap_track) &&
               !(o.write_mask & (WM_MOM | WM_EKIN | WM_ETOT));
    }
    int small_steps(int s, int i0, int i1) const {
        NdSmall P{};
        P.i0 = i0;
        P.i1 = i1;
        P.iters = iters;
        P.mask = J->o.write_mask | (acf ? (uint32_t)WM_ACF : 0u);
        P.ldx = tile_ldx(J->n, 1);
        P.hist = hist(s);
        P.hc = HC;
        P.rows_out = rows_out(s);
        return nd_small_launch<T>(S, Lc.D.logn, Lc.D, P, J->stream);
    }
    // rows i0 .. i1 of solve s
    int steps(int s, int i0, int i1) {
        if (small()) return small_steps(s, i0, i1);
        for (int i = i0; i <= i1; ++i)
            if (const int rc = step(s, i)) return rc;
        return ZQD_OK;
    }
    // this solve's wavefunction history entry of step i (write.wavefunction), or null
    cx<T>* whist(int s, int i) const {
        return J->wfn_hist.p ? J->wfn_hist.as<cx<T>>() + ((size_t)s * (iters + 1) + i) * S * J->N : nullptr;
    }
    // finalize descriptors
    NdFin fin(int s, int kind, size_t x0, size_t x1, bool k, uint32_t mask, double* row, int i) const {
        const Opts& o = J->o;
        NdFin f{};
        f.row = row;
        f.rows_out = rows_out(s);
        f.book = J->book.as<NdBook>();
        f.x0 = x0;
        f.x1 = x1;
        f.k0 = Lc.K;
        f.k1 = k ? Lc.K + Lc.k_cols : Lc.K;
        f.stop_norm = o.cap_stop_norm;
        f.mask = mask;
        f.row_index = i;
        f.kind = kind;
        f.has_stop = kind == 0 && o.has_cap && o.cap_has_stop;
        return f;
    }
    int itp_ops(int s) { // quantum_dynamics.zig:898-906
        int rc;
        for (int j = 0; j < s; ++j) {
            nd_dot_kernel<T><<<ng, 256, 0, J->stream>>>(Lc.D, j, Lc.G);
            if ((rc = Lc.reduce(Lc.G, Lc.G + ng, 2))) return rc;
            nd_orth_apply_kernel<T><<<ng, 256, 0, J->stream>>>(Lc.D, j, Lc.scal());
        }
        nd_dot_kernel<T><<<ng, 256, 0, J->stream>>>(Lc.D, -1, Lc.G);
        if ((rc = Lc.reduce(Lc.G, Lc.G + ng, 1))) return rc;
        nd_normalize_kernel<T, S><<<ng, 256, 0, J->stream>>>(Lc.D, Lc.scal(), 0, 0);
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    int prologue(int s) {
        const Opts& o = J->o;
        ZQD_CUDA(cudaMemsetAsync(J->flags.p, 0, 2 * sizeof(int), J->stream));
        ZQD_CUDA(cudaMemsetAsync(J->book.p, 0, sizeof(NdBook), J->stream));
        if (s == 0 && o.pot_td) { // a later run starts again from the t = 0 tables (Hamiltonian.init, Propagator.init)
            nd_table_kernel<T, S><<<(unsigned)((J->N + 127) / 128), 128, 0, J->stream>>>(Lc.D, 0.0, 1);
            ZQD_CUDA(cudaGetLastError());
        }
        // setGaussian, normalise, toDia, acf reference (quantum_dynamics.zig:867-882)
        nd_gauss_kernel<T><<<ng, 256, 0, J->stream>>>(Lc.D, Lc.G);
        ZQD_CUDA(cudaGetLastError());
        if (int rc = Lc.reduce(Lc.G, Lc.G + ng, 1)) return rc;
        nd_normalize_kernel<T, S><<<ng, 256, 0, J->stream>>>(Lc.D, Lc.scal(), o.ic_adiabatic ? 1 : 0, acf ? 1 : 0);
        ZQD_CUDA(cudaGetLastError());
        return ZQD_OK;
    }
    // the row pass that opens a step by itself, with the absorbed sums of its first accumAbsorbed
    int open(int s, bool track) {
        const uint32_t mode = RM_RSTART | RM_FWD | RM_STORE;
        if (!track) return Lc.row(mode, 0, Lc.R2);
        return Lc.observe(mode, 0, Lc.R2, fin(s, 2, Lc.R2, Lc.R2 + Lc.row_cols, false, 0, nullptr, 0), false);
    }
    int step(int s, int i) {
        const Opts& o = J->o;
        int rc;
        const bool logstep = o.log && ((i % o.log_interval == 0) || (i == iters));
        const uint32_t mask = o.write_mask | (logstep ? (uint32_t)WM_ALL_OBS : 0u) | (acf ? (uint32_t)WM_ACF : 0u);
        const bool needk = mask & (WM_MOM | WM_EKIN | WM_ETOT);
        const uint32_t obs = mask | ((o.has_cap && o.cap_has_stop) ? (uint32_t)WM_NORM : 0u);
        double* row = hist(s) + (size_t)i * HC;
        const bool defer = deferred(s);
        if (i > 0 && (rc = Lc.step_tiles(defer ? (uint32_t)TM_SCALE : 0u))) return rc;
        if (!split || defer) {
            uint32_t mode = RM_OBS | RM_STORE | (needk ? RM_PHI : 0u);
            if (i > 0) mode |= RM_INV | RM_REND;
            if (i < iters) mode |= RM_RSTART | RM_FWD;
            NdFin f = fin(s, 0, Lc.R0, Lc.R0 + Lc.row_cols, needk, mask, row, i);
            if (defer) f.nsum_out = Lc.scal();
            const uint32_t o2 = obs | (defer ? (uint32_t)WM_NORM : 0u);
            return Lc.observe(mode, o2, Lc.R0, f, false, false, whist(s, i));
        }
        const bool track = Lc.D.track;
        if (!o.imag_nstate && !o.pot_td) { // stop_norm alone: close step i and observe it, decide, then open the next
            const uint32_t mode = RM_OBS | RM_STORE | (i > 0 ? (uint32_t)(RM_INV | RM_REND) : 0u) | (needk ? (uint32_t)RM_PHI : 0u);
            if ((rc = Lc.observe(mode, obs, Lc.R0, fin(s, 0, Lc.R0, Lc.R0 + Lc.row_cols, needk, mask, row, i), true, false, whist(s, i))))
                return rc;
            return i < iters ? open(s, track) : ZQD_OK;
        }
        // Imaginary time, first state (nothing to orthogonalise against), no absorbing potential, after
        // step 0: the pass that closes step i also sums |psi|^2, and the next pass divides by the norm
        // as it loads psi, in place of the norm and normalisation kernels (quantum_dynamics.zig:898-906
        // with no earlier states); without a time-dependent potential that pass also records the
        // step's observables and opens step i+1.
        const bool fuse = o.imag_nstate && s == 0 && i > 0 && !o.has_cap;
        if (i > 0 && (rc = Lc.row(RM_INV | RM_REND | RM_STORE | (fuse ? (uint32_t)RM_NORM : 0u), 0, Lc.R0))) return rc;
        if (fuse) { // the norm's sum into scal[0], taken out of R0 (the observables row sums R0 too)
            if ((rc = Lc.reduce(Lc.R0, Lc.R0 + Lc.row_cols, 1, true))) return rc;
        } else if (o.imag_nstate && (rc = itp_ops(s))) {
            return rc; // every i, the initial state included
        }
        if (o.pot_td && (rc = Lc.table((double)i * o.time_step, 0))) return rc;
        // R0 holds the end-of-step sums of the row pass that closed step i (none at i = 0)
        const NdFin f = fin(s, 0, i > 0 ? Lc.R0 : Lc.R1, Lc.R1 + Lc.row_cols, needk, mask, row, i);
        // stop_norm decides before the next launch; tracked absorption's carry is replaced by that launch's sums
        const bool now = f.has_stop || track;
        if (fuse && !o.pot_td && i < iters) { // normalise, observe, and open step i+1 in one pass
            const uint32_t mode = RM_SCALE | RM_OBS | RM_RSTART | RM_FWD | RM_STORE | (needk ? (uint32_t)RM_PHI : 0u);
            return Lc.observe(mode, obs, Lc.R1, f, now, false, whist(s, i));
        }
        const uint32_t omode = RM_OBS | (needk ? (uint32_t)RM_PHI : 0u) | (fuse ? (uint32_t)(RM_SCALE | RM_STORE) : 0u);
        if ((rc = Lc.observe(omode, obs, Lc.R1, f, now, false, whist(s, i)))) return rc;
        if (i < iters) {
            if (o.pot_td && (rc = Lc.table(((double)i + 0.5) * o.time_step, 1))) return rc;
            return open(s, track);
        }
        return ZQD_OK;
    }
    int epilogue(int s) {
        int rc;
        if ((rc = Lc.flush())) return rc;
        // final Observables.init(..., log = true) (quantum_dynamics.zig:949)
        const uint32_t all = WM_ALL_OBS | (acf ? (uint32_t)WM_ACF : 0u);
        // a deferred renormalisation (the last step's) is applied here, and psi stored normalised
        const uint32_t scale = deferred(s) ? (uint32_t)(RM_SCALE | RM_STORE) : 0u;
        if ((rc = Lc.observe(RM_OBS | RM_PHI | scale, all, Lc.R1,
                             fin(s, 1, Lc.R1, Lc.R1 + Lc.row_cols, true, all, J->fin.as<double>() + (size_t)s * HC, 0), true, true)))
            return rc;
        if (s + 1 < J->nsolve) // orthw.append (quantum_dynamics.zig:586-591)
            ZQD_CUDA(cudaMemcpyAsync(J->orth.as<char>() + (size_t)s * SN, J->psi_save.p, SN, cudaMemcpyDeviceToDevice, J->stream));
        return ZQD_OK;
    }
};

// every launch of a run, in stream order (captured into a graph by ZQD_ND_RUN)
int enqueue(zqd_job* J) {
    Seq q(J);
    int rc;
    for (int s = 0; s < J->nsolve; ++s) {
        if ((rc = q.prologue(s))) return rc;
        if ((rc = q.steps(s, 0, q.iters))) return rc;
        if ((rc = q.epilogue(s))) return rc;
    }
    return ZQD_OK;
}
} // namespace

// The TMA-staged passes record a load that never landed in flags[2] (the job's buffers are
// then suspect): report it as a device error.
static int check_tma(zqd_job* J) {
    if (!J->nd_tma && !J->nd_row_tma) return ZQD_OK;
    int e = 0;
    ZQD_CUDA(cudaMemcpyAsync(&e, J->flags.as<int>() + 2, sizeof(int), cudaMemcpyDeviceToHost, J->stream));
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    J->d2h += sizeof(int);
    return e ? fail(ZQD_ERR_DEVICE, "A TMA LOAD OF AN AXIS PASS DID NOT COMPLETE WITHIN ITS WAIT BUDGET") : ZQD_OK;
}

// Rows i0..i1 of solve s (zqd_job_step), launched directly; then, if the solve ended (its last
// step, or stop_norm), its final observables.  *rows: rows of the solve's history written so far.
int ZQD_ND_STEP(zqd_job* J, int s, int i0, int i1, int* rows, int* ended) {
    Seq q(J);
    int rc;
    ZQD_CUDA(cudaEventRecord(J->ev0, J->stream));
    if (i0 == 0 && (rc = q.prologue(s))) return rc;
    if ((rc = q.steps(s, i0, i1))) return rc;
    if ((rc = q.Lc.flush())) return rc;
    // the steps first, then the copies into pageable memory (one queued behind the steps would wait
    // inside the driver, where it can hold up other threads' copies)
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    int flags[2] = {0, 0}; // stopped, rows
    ZQD_CUDA(cudaMemcpyAsync(&flags[0], J->flags.p, sizeof(int), cudaMemcpyDeviceToHost, J->stream));
    ZQD_CUDA(cudaMemcpyAsync(&flags[1], q.rows_out(s), sizeof(int), cudaMemcpyDeviceToHost, J->stream));
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    J->d2h += sizeof(flags);
    *rows = flags[1];
    *ended = flags[0] || i1 >= q.iters;
    if ((rc = check_tma(J))) return rc;
    if (*ended && (rc = q.epilogue(s))) return rc;
    ZQD_CUDA(cudaEventRecord(J->ev1, J->stream));
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    float ms = 0;
    ZQD_CUDA(cudaEventElapsedTime(&ms, J->ev0, J->ev1));
    J->last_ms += ms;
    return ZQD_OK;
}

// A run is a fixed sequence of launches: it is captured into a CUDA graph on the
// first call and the graph is replayed by every later call on the job.
int ZQD_ND_RUN(zqd_job* J) {
    if (!J->nd_use_graph) {
        ZQD_CUDA(cudaEventRecord(J->ev0, J->stream));
        const int rc = enqueue(J);
        if (rc) return rc;
        ZQD_CUDA(cudaEventRecord(J->ev1, J->stream));
        ZQD_CUDA(cudaStreamSynchronize(J->stream));
        ZQD_CUDA(cudaEventElapsedTime(&J->last_ms, J->ev0, J->ev1));
        return check_tma(J);
    }
    if (!J->nd_graph) {
        ZQD_CUDA(cudaStreamBeginCapture(J->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue(J);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(J->stream, &g);
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        ZQD_CUDA(e);
        const cudaError_t ei = cudaGraphInstantiate(&J->nd_graph, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) J->nd_graph = nullptr;
        ZQD_CUDA(ei);
    }
    ZQD_CUDA(cudaEventRecord(J->ev0, J->stream));
    ZQD_CUDA(cudaGraphLaunch(J->nd_graph, J->stream));
    ZQD_CUDA(cudaEventRecord(J->ev1, J->stream));
    ZQD_CUDA(cudaStreamSynchronize(J->stream));
    ZQD_CUDA(cudaEventElapsedTime(&J->last_ms, J->ev0, J->ev1));
    return check_tma(J);
}

} // namespace zqd
