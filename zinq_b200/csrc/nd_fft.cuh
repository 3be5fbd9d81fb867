// nd_fft.cuh -- line transforms of the TMA-staged axis passes: sixteen elements of a line per
// thread, the Stockham passes between registers and one shared-memory exchange per pass boundary.
//
// Thread i of a line (i < n/16) holds elements i + t n/16, t < 16, before and after the transform.
// A pass of radix R splits them into 16/R butterflies i' = i + b n/16 (b < 16/R), whose inputs
// i' + r n/R are the thread's elements b + r 16/R: the first pass runs on the registers as loaded,
// the last pass (span p = n/R) leaves its outputs where its inputs were, and only the boundaries
// between passes go through shared memory.  Radices up to 16 need one boundary for n = 32..256 and
// two for n = 512..4096; with eight elements a thread (radices up to 8) 128, 256 and 512 points
// need two and 1024 and 2048 points three.  A line of at most 512 points belongs to one
// warp (n/16 <= 32 threads), so its boundaries need no CTA barrier.
#pragma once

#include "cx.cuh"

namespace zqd {

// padx-style line layout: element e at e + (e >> ps), ps = log2 of the first radix.  The first
// pass writes at stride R0 = 2^ps across threads, which the padding turns into an odd stride.
template <int LOGN> struct LinePlan {
    static_assert(LOGN >= 5 && LOGN <= 12, "lines of 32 to 4096 points");
    static constexpr int n = 1 << LOGN, TPL = n / 16; // threads per line
    static constexpr int NP = LOGN <= 8 ? 2 : 3;      // passes
    __host__ __device__ static constexpr int lr(int j) { // log2 radix of pass j
        return LOGN == 5 ? (j == 0 ? 3 : 2)
             : LOGN == 6 ? 3
             : LOGN == 7 ? (j == 0 ? 4 : 3)
             : LOGN == 8 ? 4
             : LOGN == 9 ? 3
             : LOGN == 10 ? (j == 0 ? 4 : 3)
             : LOGN == 11 ? (j == 1 ? 3 : 4)
                          : 4;
    }
    __host__ __device__ static constexpr int logp(int j) { return j == 0 ? 0 : logp(j - 1) + lr(j - 1); }
    // first entry of pass j in the dense twiddle table: passes j >= 1 hold W_n^(r kk n/(p R)) at
    // [(r - 1) p + kk], (R - 1) p entries each
    __host__ __device__ static constexpr int base(int j) {
        return j <= 1 ? 0 : base(j - 1) + ((1 << lr(j - 1)) - 1) * (1 << logp(j - 1));
    }
    static constexpr int ntw = n - (1 << (LOGN == 5 || LOGN == 6 || LOGN == 9 ? 3 : 4)); // table entries
    static constexpr int ps = LOGN == 5 || LOGN == 6 || LOGN == 9 ? 3 : 4;
    static_assert((1 << ps) == n - ntw, "the table's length is n minus the first radix");
    __host__ __device__ static constexpr int pad(int e) { return e + (e >> ps); }
    // pad(i + t TPL) - pad(i) for i < TPL: exact when TPL and 2^ps divide one another
    __host__ __device__ static constexpr int pad_step(int t) { return t * TPL + ((t * TPL) >> ps); }
};

// log2 of the first radix of an n-point line (what LinePlan::ps is)
__host__ __device__ constexpr int line_ps(int logn) { return logn == 5 || logn == 6 || logn == 9 ? 3 : 4; }
// stride between the exchange lines of a CTA: the padded length, rounded up so that lines whose
// threads share a quarter warp (16-byte elements) or half warp (8-byte) start in distinct banks.
// share: lines side by side across consecutive threads (tile passes: the lines of a warp), or 0
// for lines that take consecutive threads each (row passes).
template <typename T> __host__ __device__ inline int exch_stride(int logn, int share) {
    const int n = 1 << logn, q = sizeof(cx<T>) == 16 ? 8 : 16, tpl = n / 16;
    int want; // stride mod q
    if (share) want = share >= q ? 1 : (q / share) % q;
    else want = tpl >= q ? 0 : tpl;
    int ld = n + (n >> line_ps(logn));
    while (ld % q != want) ++ld;
    return ld;
}

// Tile passes: whether a warp takes whole lines (32 / TPL of them), with no CTA barrier at a transform's
// boundaries.  Not where those lines' elements side by side are less than a 32-byte sector: from 512 points
// (256 in FP32) up a warp's loads and stores at the axis stride would be part of a sector each.  There
// neighbouring threads take the tile's neighbouring lines and the CTA waits at the boundaries.
template <typename T> __host__ __device__ constexpr bool tile_warp_lines(int logn) {
    return logn <= 9 && (512 >> logn) * sizeof(cx<T>) >= 32;
}

struct SyncWarp {
    __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
struct SyncCta {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
struct SyncBar { // a named barrier of `count` threads (whole warps)
    int id, count;
    __device__ __forceinline__ void operator()() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
};

template <typename T, int LOGN, int SIGN, int J, typename SY>
__device__ __forceinline__ void line_passes(cx<T> (&v)[16], cx<T>* __restrict__ line, int i, const Tab<T>* __restrict__ tw,
                                            const SY& sync) {
    using P = LinePlan<LOGN>;
    constexpr int LR = P::lr(J), R = 1 << LR, B = 16 / R, p = 1 << P::logp(J);
    constexpr bool LAST = J == P::NP - 1;
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int ip = i + b * P::TPL, kk = ip & (p - 1);
        cx<T> u[R];
#pragma unroll
        for (int r = 0; r < R; ++r) u[r] = v[b + r * B];
        if constexpr (J > 0) {
#pragma unroll
            for (int r = 1; r < R; ++r) u[r] = tmul<SIGN>(u[r], tw[P::base(J) + (r - 1) * p + kk]);
        }
        dft<R, SIGN, T>(u);
        if constexpr (LAST) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[b + r * B] = u[r];
        } else {
            // outputs ((i' - kk) R + kk) + r p; p is 1 or a multiple of 2^ps, so the padding of r p is constant
            cx<T>* dst = line + P::pad(((ip - kk) << LR) + kk);
#pragma unroll
            for (int r = 0; r < R; ++r) dst[J == 0 ? r : r * p + ((r * p) >> P::ps)] = u[r];
        }
    }
    if constexpr (!LAST) {
        sync();
        const cx<T>* src = line + P::pad(i);
#pragma unroll
        for (int t = 0; t < 16; ++t) v[t] = src[P::pad_step(t)];
        if constexpr (J + 1 < P::NP - 1) sync(); // the next pass writes the line again
        line_passes<T, LOGN, SIGN, J + 1>(v, line, i, tw, sync);
    }
}

// n-point transform (SIGN -1 forward, +1 inverse, unnormalised) of the thread's line, in registers
// before and after.  line: the line's exchange buffer (free to write on entry: the caller has
// synchronised the line's threads since anybody read it), still being read by the line's other
// threads on return.
template <typename T, int LOGN, int SIGN, typename SY>
__device__ __forceinline__ void line_fft(cx<T> (&v)[16], cx<T>* __restrict__ line, int i, const Tab<T>* __restrict__ tw,
                                         const SY& sync) {
    line_passes<T, LOGN, SIGN, 0>(v, line, i, tw, sync);
}

// The twiddles pass by pass (LinePlan's table, ntw entries) from the natural table w of n = 2^logn
// entries exp(-2 pi i t / n); logn outside LinePlan's range leaves out untouched.
template <typename W, int LOGN = 5> inline void dense_twiddles(int logn, const W* w, W* out) {
    if constexpr (LOGN <= 12) {
        if (logn != LOGN) return dense_twiddles<W, LOGN + 1>(logn, w, out);
        using P = LinePlan<LOGN>;
        for (int j = 1; j < P::NP; ++j) {
            const int R = 1 << P::lr(j), p = 1 << P::logp(j), step = P::n / (p * R);
            for (int r = 1; r < R; ++r)
                for (int kk = 0; kk < p; ++kk) out[P::base(j) + (r - 1) * p + kk] = w[r * kk * step];
        }
    }
}

} // namespace zqd
