// scan.cuh -- exclusive scans of computed values: the input of position i is
// in(i) (N integers, recomputed instead of stored) and its prefix goes
// straight to out(i, value, prefix), so flags, prefix and assignment arrays
// need no passes of their own.  The setup's compactions are built on it.
#pragma once
#include "common.cuh"

namespace tfb {

template <int N>
struct Counts {
    int v[N];
};

namespace scan_detail {

constexpr int kThreads = 256, kItems = 8, kTile = kThreads * kItems;
constexpr int kMidThreads = 1024;

// Exclusive prefix of one value per thread over the block (and the total).
template <int N, int kT>
__device__ __forceinline__ Counts<N> block_exclusive(const Counts<N> &mine, Counts<N> &total) {
    __shared__ int warp_tot[N][kT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Counts<N> inc = mine;
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc.v[k], o);
            if (lane >= o) inc.v[k] += y;
        }
    __syncthreads();  // warp_tot may still be read from an earlier call
    if (lane == 31)
#pragma unroll
        for (int k = 0; k < N; ++k) warp_tot[k][warp] = inc.v[k];
    __syncthreads();
    Counts<N> out;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        // every warp scans the warp totals itself
        int t = lane < kT / 32 ? warp_tot[k][lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        total.v[k] = __shfl_sync(0xffffffffu, t, kT / 32 - 1);
        const int before = __shfl_sync(0xffffffffu, t, warp > 0 ? warp - 1 : 0);
        out.v[k] = (warp > 0 ? before : 0) + inc.v[k] - mine.v[k];
    }
    return out;
}

template <int N, class In>
__global__ void __launch_bounds__(kThreads) tile_sums(int n, In in, Counts<N> *__restrict__ sums) {
    const int base = blockIdx.x * kTile + threadIdx.x;
    Counts<N> s{}, total;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int i = base + q * kThreads;
        if (i < n) {
            const Counts<N> v = in(i);
#pragma unroll
            for (int k = 0; k < N; ++k) s.v[k] += v.v[k];
        }
    }
    block_exclusive<N, kThreads>(s, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Exclusive scan of the tile sums in place (one CTA).
template <int N>
__global__ void __launch_bounds__(kMidThreads) scan_sums(int tiles, Counts<N> *__restrict__ sums) {
    Counts<N> carry{};
    for (int t0 = 0; t0 < tiles; t0 += kMidThreads) {
        const int t = t0 + threadIdx.x;
        Counts<N> v{}, total;
        if (t < tiles) v = sums[t];
        const Counts<N> p = block_exclusive<N, kMidThreads>(v, total);
        if (t < tiles) {
            Counts<N> r;
#pragma unroll
            for (int k = 0; k < N; ++k) r.v[k] = carry.v[k] + p.v[k];
            sums[t] = r;
        }
#pragma unroll
        for (int k = 0; k < N; ++k) carry.v[k] += total.v[k];
    }
}

// One tile of kT threads x kItems consecutive positions per thread.
template <int N, int kT, class In, class Out>
__device__ __forceinline__ void scan_tile(int first, int n, const In &in, const Out &out, Counts<N> &carry) {
    const int base = first + static_cast<int>(threadIdx.x) * kItems;
    Counts<N> v[kItems], s{}, total;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        v[q] = Counts<N>{};
        if (base + q < n) v[q] = in(base + q);
#pragma unroll
        for (int k = 0; k < N; ++k) s.v[k] += v[q].v[k];
    }
    Counts<N> p = block_exclusive<N, kT>(s, total);
#pragma unroll
    for (int k = 0; k < N; ++k) p.v[k] += carry.v[k];
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        if (base + q < n) out(base + q, v[q], p);
#pragma unroll
        for (int k = 0; k < N; ++k) p.v[k] += v[q].v[k];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) carry.v[k] += total.v[k];
}

template <int N, class In, class Out>
__global__ void __launch_bounds__(kThreads) scan_tiles(int n, In in, Out out, const Counts<N> *__restrict__ sums) {
    Counts<N> carry = sums[blockIdx.x];
    scan_tile<N, kThreads>(blockIdx.x * kTile, n, in, out, carry);
}

template <int N, class In, class Out>
__global__ void __launch_bounds__(kMidThreads) scan_one_cta(int n, In in, Out out) {
    Counts<N> carry{};
    for (int first = 0; first < n; first += kMidThreads * kItems)
        scan_tile<N, kMidThreads>(first, n, in, out, carry);
}

}  // namespace scan_detail

// out(i, in(i), sum of in(j), j < i) for i in [0, n).  in is evaluated twice
// per position and must not depend on what out writes.  Up to 16,384
// positions one CTA does it in one launch (two rounds of its 8,192; a launch
// costs 2 us, a round under 1 us); larger scans take three launches.
template <int N, class In, class Out>
void scan_apply(tf_ctx *ctx, int n, const In &in, const Out &out, const char *name) {
    using namespace scan_detail;
    if (n <= 0) return;
    if (n <= 2 * kMidThreads * kItems) {
        scan_one_cta<N><<<1, kMidThreads, 0, ctx->stream>>>(n, in, out);
        launched(ctx, name);
        return;
    }
    const int tiles = static_cast<int>((static_cast<int64_t>(n) + kTile - 1) / kTile);
    TempBuffer<Counts<N>> sums(ctx, static_cast<size_t>(tiles));
    tile_sums<N><<<tiles, kThreads, 0, ctx->stream>>>(n, in, sums.data());
    launched(ctx, name);
    scan_sums<N><<<1, kMidThreads, 0, ctx->stream>>>(tiles, sums.data());
    launched(ctx, name);
    scan_tiles<N><<<tiles, kThreads, 0, ctx->stream>>>(n, in, out, sums.data());
    launched(ctx, name);
}

}  // namespace tfb
