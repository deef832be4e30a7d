// setup.cu -- device stages of the aggregation AMG setup: canonical form,
// strength graph, synchronous handshake matching, graph contraction,
// singleton absorption, member tables and the Galerkin product.
//
// The algorithm is the reference's (src/Multigrid/GpuAggregation.cu, whose
// host statement is test/support/NativeAggregationOracle.cu); the results
// (aggregates, member order, histograms, coarse sparsity) are meant to be
// bit-identical to it, which is why every stage keeps the reference's
// snapshot semantics: proposals of a matching round are all written before
// any are accepted, and absorption accepts from one snapshot of proposals.
// Rows are handled by themselves wherever a stage allows it: strength weights
// lie on the operator's own pattern, the Galerkin product merges the rows of an
// aggregate, aggregates are numbered by scans (scan.cuh), and their members are
// sorted in place (at most four).  The sort over all coordinates (sort.cu) is
// left for unsymmetric strength graphs, merged rows of more than 512 entries
// and operators that arrive unsorted.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "scan.cuh"
#include "setup.cuh"

namespace tfb {
namespace {

template <class T>
using Temp = TempBuffer<T>;

__device__ __forceinline__ uint64_t sort_key(int r, int c, int bits) {
    return (static_cast<uint64_t>(static_cast<unsigned>(r)) << bits) | static_cast<unsigned>(c);
}

// Symmetric edge priority (GpuAggregation.cu:49-54): splitmix64 finaliser of
// (min(i,j) << 32 | max(i,j)); breaks equal-weight proposals identically on
// both endpoints.
__device__ __forceinline__ uint64_t edge_priority(int i, int j) {
    uint64_t h = (static_cast<uint64_t>(static_cast<unsigned>(min(i, j))) << 32) | static_cast<unsigned>(max(i, j));
    h = (h ^ (h >> 30)) * 0xbf58476d1ce4e5b9ULL;
    h = (h ^ (h >> 27)) * 0x94d049bb133111ebULL;
    return h ^ (h >> 31);
}

// Coordinate keys of every entry, optionally mapped (canonical: map null;
// Galerkin: map = aggregates).  GpuAggregation.cu:136-146.
__global__ void map_entries(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                            const double *__restrict__ a, const int32_t *__restrict__ map, uint64_t *__restrict__ keys,
                            double *__restrict__ vals, int bits) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = map ? map[i] : i;
    for (int32_t j = rp[i]; j < rp[i + 1]; ++j) {
        const int c = map ? map[ci[j]] : ci[j];
        keys[j] = sort_key(r, c, bits);
        vals[j] = a[j];
    }
}

// Strong edges in both directions (GpuAggregation.cu:339-364); count pass
// when keys is null, fill pass at the scanned offsets otherwise.
__global__ void strength_edges(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                               const double *__restrict__ a, const double *__restrict__ mx, double theta,
                               uint64_t *__restrict__ keys, double *__restrict__ w, int32_t *__restrict__ count,
                               int bits) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int pos = keys ? count[i] : 0;
    const double m = mx[i];
    for (int32_t j = rp[i]; j < rp[i + 1]; ++j) {
        const int c = ci[j];
        const double weight = (i != c && m > 0 && fabs(a[j]) / m >= theta) ? fabs(a[j]) / m : 0.0;
        if (weight > 0) {
            if (keys) {
                keys[pos] = sort_key(i, c, bits);
                keys[pos + 1] = sort_key(c, i, bits);
                w[pos] = w[pos + 1] = weight;
            }
            pos += 2;
        }
    }
    if (!keys) count[i] = pos;
}

// A level's arrays from its native operator in one pass: the structure and the
// values in their storage V, the inverse diagonal in the iteration precision S
// (inverse_diagonal's expression), columns as row offsets, the largest
// |off-diagonal| of each row and the checks (row_stats, inverse_diagonal,
// delta_columns).  kG lanes share a row.  Bytes bound it on the finest level
// (read once: 12 B an entry, written 10-14 B); on the others its launch does,
// which is why one pass and one read-back of the flags took the place of six
// launches and three read-backs a level.  Whole setup, with the copies' sizes
// from one pass (copy_shapes): 2.1M rows FP32 8.9 -> 7.8 ms, a graph of 60k
// rows 6.4 -> 5.5 ms.
template <int kG, class S, class V>
__global__ void level_arrays_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                    const double *__restrict__ a, LevelArrays<S, V> out, int *flags) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t i64 = t / kG;
    const int lane = static_cast<int>(t % kG);
    int found = 0;
    if (i64 < n) {
        const int i = static_cast<int>(i64);
        const int32_t begin = rp[i], end = rp[i + 1];
        if (lane == 0) {
            out.rp[i] = begin;
            if (i == n - 1) out.rp[n] = end;
        }
        double diag = 0, mx = 0;
        S d = S(0);
        for (int32_t j = begin + lane; j < end; j += kG) {
            const double v = a[j];
            const int c = ci[j];
            const V stored = static_cast<V>(v);
            out.ci[j] = c;
            out.val[j] = stored;
            if (!isfinite(v)) found |= kLevelInvalid;
            if (c == i) {
                diag = v;
                d += stored;
            } else {
                mx = fmax(mx, fabs(v));
            }
            if (out.cd) {
                const int o = c - i;
                if (o < -32767 || o > 32767) found |= kLevelWide;
                else out.cd[j] = static_cast<int16_t>(o);
            }
        }
        // (one lane holds the diagonal, the others 0)
        const unsigned group = (kG == 32 ? 0xffffffffu : ((1u << (kG & 31)) - 1u)) << ((threadIdx.x & 31) / kG * kG);
#pragma unroll
        for (int o = kG / 2; o > 0; o >>= 1) {
            mx = fmax(mx, __shfl_xor_sync(group, mx, o));
            diag += __shfl_xor_sync(group, diag, o);
            d += __shfl_xor_sync(group, d, o);
        }
        if (lane == 0) {
            if (diag == 0 || !isfinite(diag) || !isfinite(1.0 / diag)) found |= kLevelInvalid;
            const S inv = S(1) / d;
            if (!isfinite(d) || d == S(0) || !isfinite(inv)) found |= kLevelDiagonal;
            out.dinv[i] = inv;
            out.row_max[i] = mx;
        }
    }
    found = __reduce_or_sync(0xffffffffu, found);
    if ((threadIdx.x & 31) == 0 && (found & ~*flags)) atomicOr(flags, found);
}

// Strength weights on the operator's own pattern: w[j] is the weight of edge
// (i, c), the larger of its two directions' (GpuAggregation.cu:339-390), and
// 0 where neither is strong and on the diagonal.  Such a graph needs no
// sort, reduction and compaction of its own; the stages that read it skip
// weights of 0.  flags: bit 0 some edge is strong, bit 1 a strong edge has no
// entry for its other direction (then only the sorted graph holds it).
// kG lanes share a row; the other direction is found by bisection in row c.
template <int kG>
__global__ void strength_weights_kernel(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                        const double *__restrict__ a, const double *__restrict__ mx, double theta,
                                        double *__restrict__ w, int *flags) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t i64 = t / kG;
    int found = 0;
    if (i64 < n) {
        const int i = static_cast<int>(i64);
        auto strong = [&](double v, double m) {
            const double s = m > 0 ? fabs(v) / m : 0.0;
            return m > 0 && s >= theta ? s : 0.0;
        };
        const double m = mx[i];
        const int32_t end = rp[i + 1];
        for (int32_t j = rp[i] + static_cast<int32_t>(t % kG); j < end; j += kG) {
            const int c = ci[j];
            double s = 0;
            if (c != i) {
                s = strong(a[j], m);
                int32_t lo = rp[c], hi = rp[c + 1];
                const int32_t last = hi;
                while (lo < hi) {
                    const int32_t mid = (lo + hi) >> 1;
                    if (ci[mid] < i) lo = mid + 1;
                    else hi = mid;
                }
                if (lo < last && ci[lo] == i) s = fmax(s, strong(a[lo], mx[c]));
                else if (s > 0) found |= 2;
                if (s > 0) found |= 1;
            }
            w[j] = s;
        }
    }
    found = __reduce_or_sync(0xffffffffu, found);
    if ((threadIdx.x & 31) == 0 && (found & ~*flags)) atomicOr(flags, found);
}

// The vertices of a matching: the rows themselves, or pairs of rows (lo, hi;
// hi < 0 for a single row) with map giving the pair of every row.  The graph
// over pairs is never formed: a pair's edges are its rows' edges seen through
// map, and a proposal (the best edge to an unmatched vertex) comes out the
// same whether parallel edges are merged by their maximum first or not.
struct Vertices {
    const int32_t *lo{nullptr}, *hi{nullptr}, *map{nullptr};
    const int32_t *count{nullptr};  // their number, when the host does not know it
    int n{0};                       // their number, or a bound of it
    __device__ __forceinline__ int size() const { return count ? *count : n; }
    __device__ __forceinline__ int of(int row) const { return map ? map[row] : row; }
};

// A handshake matching in progress.  Round r works on the vertices still
// open after round r - 1 (open[r & 1], their number in counts[r]; all of them
// in round 0, which has no list): most vertices are matched after two rounds.
// The order of a list is arbitrary and decides nothing.
struct Matching {
    Vertices vs;
    const int32_t *rp, *ci;
    const double *w;
    int32_t *mate;      // -1: unmatched
    uint8_t *taken;     // mate[v] >= 0, one byte for the proposals' gathers
    int32_t *proposal;  // of the vertices open in the round
    int32_t *open[2];
    int32_t *counts;
    __device__ __forceinline__ int size(int round) const { return round ? counts[round] : vs.size(); }
    __device__ __forceinline__ int at(int round, int k) const { return round ? open[round & 1][k] : k; }
};

// (s, c) beats (score, best) as v's proposal (GpuAggregation.cu:402-431):
// larger weight, then larger edge priority, then smaller vertex.
__device__ __forceinline__ bool better(int v, double s, int c, double score, int best) {
    if (s != score) return s > score;
    if (c < 0 || c == best) return false;
    if (best < 0) return s > 0;
    const uint64_t a = edge_priority(v, c), b = edge_priority(v, best);
    return a > b || (a == b && c < best);
}

// The proposal of open vertex v (v < 0: none), its best unmatched neighbour,
// by kG consecutive lanes of a full warp; valid in each of them.  Two entries
// of a lane are in flight; only an edge that would win asks whether its
// neighbour is taken, and in the first round nobody is.
template <int kG>
__device__ __forceinline__ int propose(const Matching &m, int v, int lane, bool first) {
    int best = -1;
    double score = 0;
    auto consider = [&](double s, int32_t column) {
        if (!(s > 0) || s < score) return;
        const int c = m.vs.of(column);
        if (c == v || !better(v, s, c, score, best) || (!first && m.taken[c])) return;
        best = c;
        score = s;
    };
    for (int part = 0; part < 2 && v >= 0; ++part) {
        const int row = m.vs.lo ? (part ? m.vs.hi[v] : m.vs.lo[v]) : (part ? -1 : v);
        if (row < 0) break;
        const int32_t end = m.rp[row + 1];
        for (int32_t j = m.rp[row] + lane; j < end; j += 2 * kG) {
            const bool two = j + kG < end;
            const double s0 = m.w[j], s1 = two ? m.w[j + kG] : 0.0;
            const int c0 = m.ci[j], c1 = two ? m.ci[j + kG] : 0;
            consider(s0, c0);
            consider(s1, c1);
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = kG / 2; o > 0; o >>= 1) {
        const double s = __shfl_xor_sync(0xffffffffu, score, o);
        const int c = __shfl_xor_sync(0xffffffffu, best, o);
        if (better(v, s, c, score, best)) {
            best = c;
            score = s;
        }
    }
    return best;
}

// Proposals of one round, from one snapshot of the matching
// (GpuAggregation.cu:402-431).  Bound: reading the rows of the open vertices.
// 128^3 (2.1M rows, ncu): all proposals of a setup 1,487 us, 1,795 us with one
// entry of a lane in flight; the finest level's first eight rounds took 980 us
// when they visited every vertex, now 246 us and 138 us of acceptances.
template <int kG>
__global__ void __launch_bounds__(kBlock) match_propose(const __grid_constant__ Matching m, int round) {
    const int n = m.size(round), lane = threadIdx.x & 31;
    const int64_t step = static_cast<int64_t>(gridDim.x) * (kBlock / kG);
    for (int64_t k0 = (blockIdx.x * static_cast<int64_t>(kBlock) + threadIdx.x - lane) / kG; k0 < n; k0 += step) {
        const int64_t k = k0 + lane / kG;
        const int v = k < n ? m.at(round, static_cast<int>(k)) : -1;
        const int p = propose<kG>(m, v, lane % kG, round == 0);
        if (v >= 0 && lane % kG == 0) m.proposal[v] = p;
    }
}

// Mutual proposals become pairs (GpuAggregation.cu:440-449); the others that
// proposed at all stay open (a vertex without a proposal never gets one).
__device__ __forceinline__ void accept_one(const Matching &m, int round, int v) {
    bool stays = false;
    if (v >= 0) {
        const int p = m.proposal[v];
        if (p >= 0) {
            stays = m.proposal[p] != v;
            if (!stays) {
                m.mate[v] = p;
                m.taken[v] = 1;
            }
        }
    }
    const unsigned all = __ballot_sync(0xffffffffu, stays);
    if (!all) return;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0) base = atomicAdd(m.counts + round + 1, __popc(all));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (stays) m.open[(round + 1) & 1][base + __popc(all & ((1u << lane) - 1u))] = v;
}

__global__ void __launch_bounds__(kBlock) match_accept(const __grid_constant__ Matching m, int round) {
    const int n = m.size(round), lane = threadIdx.x & 31;
    const int64_t step = static_cast<int64_t>(gridDim.x) * kBlock;
    for (int64_t k0 = blockIdx.x * static_cast<int64_t>(kBlock) + threadIdx.x - lane; k0 < n; k0 += step)
        accept_one(m, round, k0 + lane < n ? m.at(round, static_cast<int>(k0) + lane) : -1);
}

// Scan input: 1 for the vertex that stands for its pair (or itself alone).
struct RootFlag {
    Vertices vs;
    const int32_t *mate;
    __device__ Counts<1> operator()(int v) const {
        if (v >= vs.size()) return {0};
        const int m = mate[v];
        return {m < 0 || v < m ? 1 : 0};
    }
};

// Scan output over the rows' matching: pair k = (lo, hi), map of its rows;
// position n carries the number of pairs.
struct AssignPairs {
    RootFlag f;
    int32_t *lo, *hi, *map, *count;
    __device__ void operator()(int v, const Counts<1> &flag, const Counts<1> &before) const {
        const int k = before.v[0];
        if (v == f.vs.n) *count = k;
        if (!flag.v[0]) return;
        const int m = f.mate[v];
        if (lo) {
            lo[k] = v;
            hi[k] = m;
        }
        map[v] = k;
        if (m >= 0) map[m] = k;
    }
};

// Scan output over the pairs' matching: the rows of aggregate k (at most
// four), its size and the map of its rows.
struct AssignAggregates {
    RootFlag f;
    int32_t *slots, *sizes, *map, *count;
    __device__ void operator()(int v, const Counts<1> &flag, const Counts<1> &before) const {
        const int k = before.v[0];
        if (v == f.vs.n) *count = k;
        if (!flag.v[0]) return;
        int size = 0;
        auto add = [&](int row) {
            if (row < 0) return;
            slots[static_cast<int64_t>(k) * 4 + size++] = row;
            map[row] = k;
        };
        const int m = f.mate[v];
        add(f.vs.lo[v]);
        add(f.vs.hi[v]);
        if (m >= 0) {
            add(f.vs.lo[m]);
            add(f.vs.hi[m]);
        }
        sizes[k] = size;
    }
};

// Cross-aggregate edges of the graph under map (GpuAggregation.cu:534-553).
__global__ void map_graph(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                          const double *__restrict__ w, const int32_t *__restrict__ map, int32_t *__restrict__ offsets,
                          uint64_t *__restrict__ keys, double *__restrict__ vals, int bits) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int pos = keys ? offsets[i] : 0;
    const int mi = map[i];
    for (int32_t j = rp[i]; j < rp[i + 1]; ++j) {
        const int mc = map[ci[j]];
        if (mi != mc && w[j] > 0) {
            if (keys) {
                keys[pos] = sort_key(mi, mc, bits);
                vals[pos] = w[j];
            }
            ++pos;
        }
    }
    if (!keys) offsets[i] = pos;
}

// A singleton proposes to the neighbouring aggregate of size 2..3 with the
// largest weight, ties to the smaller aggregate id (GpuAggregation.cu:646-669).
struct Absorption {
    const int32_t *rp, *ci;
    const double *w;
    const int32_t *count;  // aggregates
    int32_t *map, *sizes, *slots, *proposal;
    double *scores;
};

// The lanes of this thread's group of kG.
template <int kG>
__device__ __forceinline__ unsigned group_mask() {
    return (kG == 32 ? 0xffffffffu : ((1u << (kG & 31)) - 1u)) << ((threadIdx.x & 31) / kG * kG);
}

__device__ __forceinline__ bool proposes(const Absorption &a, int i) {
    return a.sizes[a.map[i]] == 1;  // (nobody writes sizes while proposals are made)
}

// The proposal of singleton i by kG consecutive lanes.
template <int kG>
__device__ __forceinline__ void propose_absorption(const Absorption &a, int i, int lane) {
    const auto [rp, ci, w, count, map, sizes, slots, proposal, scores] = a;
    int best = -1;
    double score = 0;
#pragma unroll 2
    for (int32_t j = rp[i] + lane; j < rp[i + 1]; j += kG) {
        const double s = w[j];
        if (s <= 0 || s < score) continue;
        const int c = map[ci[j]];
        if (sizes[c] < 2 || sizes[c] >= 4) continue;
        if (s > score || (s == score && (best < 0 || c < best))) {
            best = c;
            score = s;
        }
    }
    __syncwarp(group_mask<kG>());
#pragma unroll
    for (int o = kG / 2; o > 0; o >>= 1) {
        const double s = __shfl_xor_sync(group_mask<kG>(), score, o);
        const int c = __shfl_xor_sync(group_mask<kG>(), best, o);
        if (c >= 0 && (s > score || (s == score && (best < 0 || c < best)))) {
            best = c;
            score = s;
        }
    }
    if (lane == 0) {
        proposal[i] = best;
        scores[i] = score;
    }
}

// Each target keeps its best distinct proposers, weight descending then
// fine id ascending, up to its remaining capacity (GpuAggregation.cu:685-720),
// and takes them in: map, slots and sizes are updated in place.  kG lanes
// share aggregate c and its rows' entries; each keeps its best two and the
// lanes merge them.  A group reads only its own aggregate's size and slots (a
// singleton's size may turn from 1 to 0 under its own group, which has
// nothing to do either way), and the proposals of the kernel before.
// Bound by the latency of one row after another: a lane per row and aggregate
// (8 + 8 launches of a 60k-row graph setup) took 444 + 155 us, and that setup
// 5.47 ms; lanes by the mean row length 4.93 ms.
__device__ __forceinline__ bool accepts(const Absorption &a, int c) {
    return c < *a.count && a.sizes[c] >= 2 && a.sizes[c] < 4;
}

template <int kG>
__device__ __forceinline__ void accept_absorption(const Absorption &a, int c, int lane) {
    const auto [rp, ci, w, count, map, sizes, slots, proposal, scores] = a;
    const int size = sizes[c];
    int s0 = -1, s1 = -1;  // best and second proposer
    double w0 = -1, w1 = -1;
    auto offer = [&](int i, double s) {
        if (i < 0 || i == s0 || i == s1) return;
        if (s > w0 || (s == w0 && i < s0)) {
            s1 = s0;
            w1 = w0;
            s0 = i;
            w0 = s;
        } else if (s > w1 || (s == w1 && i < s1)) {
            s1 = i;
            w1 = s;
        }
    };
    for (int k = 0; k < size; ++k) {
        const int row = slots[static_cast<int64_t>(c) * 4 + k];
#pragma unroll 2
        for (int32_t j = rp[row] + lane; j < rp[row + 1]; j += kG) {
            const int i = ci[j];
            if (proposal[i] == c) offer(i, scores[i]);
        }
    }
    __syncwarp(group_mask<kG>());
#pragma unroll
    for (int o = kG / 2; o > 0; o >>= 1) {
        const int i0 = __shfl_xor_sync(group_mask<kG>(), s0, o), i1 = __shfl_xor_sync(group_mask<kG>(), s1, o);
        const double v0 = __shfl_xor_sync(group_mask<kG>(), w0, o), v1 = __shfl_xor_sync(group_mask<kG>(), w1, o);
        offer(i0, v0);
        offer(i1, v1);
    }
    if (lane != 0) return;
    int now = size;
    for (const int i : {s0, size == 2 ? s1 : -1}) {
        if (i < 0) continue;
        sizes[map[i]] = 0;
        map[i] = c;
        slots[static_cast<int64_t>(c) * 4 + now++] = i;
    }
    if (now != size) sizes[c] = now;
}

// One thread looks at each row; the singletons are listed per warp, and kG
// lanes share one of the list: with kG lanes on every row most of them waited
// on gathers for rows of other aggregates (heat operator of 2.1M rows, twelve
// launches: 305 -> 162 us).  Whole warps (long rows) have no list, a warp
// would go through it alone.  Aggregates with room are too many of all for a
// list to pay (329 us without, 372 us with one).
template <int kG>
__global__ void __launch_bounds__(kBlock) propose_absorption_kernel(int n, const __grid_constant__ Absorption a) {
    constexpr int kLook = kG == 32 ? 32 : 1;  // lanes that look at a row
    __shared__ int list[kBlock];
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int i = static_cast<int>(t / kLook), lane = threadIdx.x & 31;
    const bool mine = t / kLook < n && proposes(a, i);
    if (t / kLook < n && !mine) a.proposal[i] = -1;
    if constexpr (kG == 32) {
        if (mine) propose_absorption<kG>(a, i, lane);
    } else {
        const unsigned all = __ballot_sync(0xffffffffu, mine);
        int *of_warp = list + (threadIdx.x - lane);
        if (mine) of_warp[__popc(all & ((1u << lane) - 1u))] = i;
        __syncwarp();
        for (int k = lane / kG; k < __popc(all); k += 32 / kG) propose_absorption<kG>(a, of_warp[k], lane % kG);
    }
}
template <int kG>
__global__ void __launch_bounds__(kBlock) accept_absorption_kernel(int n, const __grid_constant__ Absorption a) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int c = static_cast<int>(t / kG);
    if (t / kG < n && accepts(a, c)) accept_absorption<kG>(a, c, static_cast<int>(t % kG));
}

// Scan input: the aggregate counted under its size, 1 to 4 rows (an emptied
// one nowhere).  The four counts give the number of aggregates and of rows
// before one, and at the end the histogram.
struct SizeOf {
    const int32_t *sizes, *count;
    __device__ Counts<4> operator()(int c) const {
        const int s = c < *count ? sizes[c] : 0;
        return {{s == 1, s == 2, s == 3, s == 4}};
    }
};

// Scan output: emptied aggregates closed up (GpuAggregation.cu:745-757), the
// members of each in ascending order and the map; position `bound` carries
// the totals.
struct PackAggregates {
    int bound;
    const int32_t *slots;
    int32_t *off, *mem, *map, *coarse, *histogram;
    const int *strength_flags;  // handed on to the read-back (may be null)
    int32_t *flags;
    __device__ void operator()(int c, const Counts<4> &v, const Counts<4> &before) const {
        const auto &b = before.v;
        const int k = b[0] + b[1] + b[2] + b[3], to = b[0] + 2 * b[1] + 3 * b[2] + 4 * b[3];
        const int size = v.v[0] + 2 * v.v[1] + 3 * v.v[2] + 4 * v.v[3];
        if (c == bound) {
            *coarse = k;
            off[k] = to;
            for (int q = 0; q < 4; ++q) histogram[q] = b[q];
            *flags = strength_flags ? *strength_flags : 0;
        }
        if (!size) return;
        int32_t m[4] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int32_t row = q < size ? slots[static_cast<int64_t>(c) * 4 + q] : INT_MAX;
#pragma unroll
            for (int r = 0; r <= q; ++r) {  // insertion into the sorted m[0..q)
                const int32_t low = min(m[r], row);
                row = max(m[r], row);
                m[r] = low;
            }
        }
        off[k] = to;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < size) {
                mem[to + q] = m[q];
                map[m[q]] = k;
            }
    }
};

// ---- Galerkin product by rows ----
//
// Aggregates have at most four members, so row r of P^T A P holds the mapped
// entries of at most four rows of A: a warp sorts them among themselves in
// registers instead of a radix sort over the coordinates of the whole matrix
// (five passes of 32 bytes per entry on 128^3).

// Entries of the member rows of every aggregate (zero at coarse) and their
// largest number.
__global__ void merged_lengths(int coarse, const int32_t *__restrict__ off, const int32_t *__restrict__ mem,
                               const int32_t *__restrict__ rp, int32_t *__restrict__ len, int *longest) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    int n = 0;
    if (c < coarse)
        for (int32_t k = off[c]; k < off[c + 1]; ++k) n += rp[mem[k] + 1] - rp[mem[k]];
    if (c <= coarse) len[c] = n;
    for (int o = 16; o > 0; o >>= 1) n = max(n, __shfl_xor_sync(0xffffffffu, n, o));
    if ((threadIdx.x & 31) == 0 && n > *longest) atomicMax(longest, n);
}

// Sorts 32 K keys held by a warp, element lane * K + r in k[r] (bitonic).
template <int K, class Key>
__device__ __forceinline__ void warp_sort(Key (&k)[K], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= K) {
                const int lx = stride / K;
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    const Key other = __shfl_xor_sync(0xffffffffu, k[r], lx);
                    const bool up = ((lane * K + r) & size) == 0, lower = (lane & lx) == 0;
                    k[r] = (up == lower) == (k[r] < other) ? k[r] : other;
                }
            } else {
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    if (r & stride) continue;
                    const bool up = ((lane * K + r) & size) == 0;
                    const Key a = k[r], b = k[r | stride];
                    const bool swap = up == (a > b);
                    k[r] = swap ? b : a;
                    k[r | stride] = swap ? a : b;
                }
            }
        }
    }
}

// Longest merged row of merge_rows: 512 entries of 14 bytes in shared memory
// for each of four warps.  Longer ones take the sort over all coordinates.
constexpr int kMergeMax = 512;
// Bits of an entry's position in a merged row of at most 32 kMax entries.
constexpr int merge_seq_bits(int kMax) { return kMax <= 1 ? 5 : 1 + merge_seq_bits(kMax / 2); }

// The entries of one coarse row: entry q < n is entry q + shift of A.
struct MergeSpan {
    int p1, p2, p3, n, s0, s1, s2, s3;
    __device__ __forceinline__ int entry(int q) const {
        return q + (q < p1 ? s0 : (q < p2 ? s1 : (q < p3 ? s2 : s3)));
    }
};

// Merges a span of at most 32 K entries; returns the row's length (lane 31).
template <int K, int kSeqBits, class Key>
__device__ __forceinline__ int merge_row(const MergeSpan &m, const int32_t *__restrict__ ci,
                                         const double *__restrict__ a, const int32_t *__restrict__ map, int lane,
                                         double *val, int32_t *col, uint16_t *seq, int32_t *__restrict__ tcol,
                                         double *__restrict__ tval) {
    constexpr unsigned kSeq = (1u << kSeqBits) - 1u;
    Key key[K];
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const int q = r * 32 + lane;
        key[r] = static_cast<Key>(~Key(0));
        if (q < m.n) {
            const int j = m.entry(q);
            key[r] = (static_cast<Key>(static_cast<unsigned>(map[ci[j]])) << kSeqBits) | static_cast<unsigned>(q);
            val[q] = a[j];
        }
    }
    warp_sort<K>(key, lane);
    const Key before = __shfl_up_sync(0xffffffffu, key[K - 1], 1);
    unsigned heads = 0;
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const int e = lane * K + r;
        if (e < m.n) {
            const int32_t mine = static_cast<int32_t>(key[r] >> kSeqBits);
            col[e] = mine;
            seq[e] = static_cast<uint16_t>(key[r] & kSeq);
            const Key left = r > 0 ? key[r > 0 ? r - 1 : 0] : before;
            if (e == 0 || static_cast<int32_t>(left >> kSeqBits) != mine) heads |= 1u << r;
        }
    }
    __syncwarp();
    int inc = __popc(heads);
    const int own = inc;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    int out = inc - own;
#pragma unroll
    for (int r = 0; r < K; ++r) {
        if (!(heads >> r & 1u)) continue;
        const int e = lane * K + r;
        const int32_t mine = col[e];
        double sum = val[seq[e]];
        for (int q = e + 1; q < m.n && col[q] == mine; ++q) sum += val[seq[q]];
        tcol[out] = mine;
        tval[out] = sum;
        ++out;
    }
    return inc;
}

// Row c of P^T A P (one warp): its members' entries (col = map[ci], in member
// and entry order) sorted by (column, that order); each run of a column is
// then added left to right, the order in which the stable sort over all
// coordinates adds it, so the sums are the same bits.  The row goes to
// tcol/tval from base[c], its length to count[c].
//
// Bound: the sort's instructions, not memory.  Each row is sorted in the
// smallest power of two that holds it (kMax: the level's longest row), with
// 32-bit keys where the coarse column and the position fit one.  128^3 (ncu):
// finest level, 598k rows of 24 entries, 0.28 ms; the other eight levels
// together 0.22 ms, 0.39 ms with every row sorted as the longest.  Map, sort,
// reduce and unpack took 3.4 ms on the finest level.
template <int kMax, int kWarps, class Key>
__global__ void __launch_bounds__(kWarps * 32) merge_rows(int coarse, const int32_t *__restrict__ off,
                                                          const int32_t *__restrict__ mem,
                                                          const int32_t *__restrict__ rp,
                                                          const int32_t *__restrict__ ci,
                                                          const double *__restrict__ a,
                                                          const int32_t *__restrict__ map,
                                                          const int32_t *__restrict__ base, int32_t *__restrict__ tcol,
                                                          double *__restrict__ tval, int32_t *__restrict__ count) {
    constexpr int kCap = 32 * kMax;
    __shared__ double s_val[kWarps][kCap];
    __shared__ int32_t s_col[kWarps][kCap];
    __shared__ uint16_t s_seq[kWarps][kCap];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * kWarps + warp;
    if (c >= coarse) {
        if (c == coarse && lane == 0) count[c] = 0;  // the scan's sentinel
        return;
    }
    const int o0 = off[c], members = off[c + 1] - o0;
    int start = 0, len = 0;
    if (lane < members) {
        const int row = mem[o0 + lane];
        start = rp[row];
        len = rp[row + 1] - start;
    }
    MergeSpan m;
    m.p1 = __shfl_sync(0xffffffffu, len, 0);
    m.p2 = m.p1 + __shfl_sync(0xffffffffu, len, 1);
    m.p3 = m.p2 + __shfl_sync(0xffffffffu, len, 2);
    m.n = m.p3 + __shfl_sync(0xffffffffu, len, 3);
    m.s0 = __shfl_sync(0xffffffffu, start, 0);
    m.s1 = __shfl_sync(0xffffffffu, start, 1) - m.p1;
    m.s2 = __shfl_sync(0xffffffffu, start, 2) - m.p2;
    m.s3 = __shfl_sync(0xffffffffu, start, 3) - m.p3;
    auto merge = [&](auto k) {
        constexpr int K = decltype(k)::value;
        const int32_t to = base[c];
        const int n = merge_row<K, merge_seq_bits(kMax), Key>(m, ci, a, map, lane, s_val[warp], s_col[warp], s_seq[warp], tcol + to,
                                        tval + to);
        if (lane == 31) count[c] = n;
    };
    if (m.n <= 32) return merge(std::integral_constant<int, 1>{});
    if constexpr (kMax >= 2)
        if (m.n <= 64) return merge(std::integral_constant<int, 2>{});
    if constexpr (kMax >= 4)
        if (m.n <= 128) return merge(std::integral_constant<int, 4>{});
    if constexpr (kMax >= 8)
        if (m.n <= 256) return merge(std::integral_constant<int, 8>{});
    if constexpr (kMax >= 16) merge(std::integral_constant<int, 16>{});
}

// The merged rows moved together: row c's entries from base[c] to rp[c]
// (eight lanes per row).
__global__ void pack_rows(int rows, const int32_t *__restrict__ base, const int32_t *__restrict__ rp,
                          const int32_t *__restrict__ tcol, const double *__restrict__ tval, int32_t *__restrict__ ci,
                          double *__restrict__ val) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t c = t >> 3;
    if (c >= rows) return;
    const int32_t to = rp[c], n = rp[c + 1] - to, from = base[c];
    for (int32_t k = static_cast<int32_t>(t & 7); k < n; k += 8) {
        ci[to + k] = tcol[from + k];
        val[to + k] = tval[from + k];
    }
}

// Calls f with the lanes that share a row, by the mean row length: a lane
// walks two or three entries of a short row (four lanes on 7-point rows read
// whole sectors), 32 lanes take rows of 24 entries or more.
template <class F>
void with_row_lanes(const Csr<double, int32_t> &a, F &&f) {
    const int64_t mean = a.nnz / a.rows;
    if (mean < 4) f(std::integral_constant<int, 1>{});
    else if (mean < 24) f(std::integral_constant<int, 4>{});
    else f(std::integral_constant<int, 32>{});
}

// Every stage of an aggregation, for the launches below and the one-CTA
// kernel.
struct AggregateState {
    int n, rounds;
    bool absorb;
    Matching rows, pairs;
    AssignPairs to_pairs;
    AssignAggregates to_aggregates;
    Absorption absorption;
    SizeOf size_of;
    PackAggregates pack;
};

// One CTA runs the whole aggregation of a small level: at 2 us and more per
// dependent launch, 45 launches cost more than one SM's work on a few
// thousand rows.  Its stages are separated by __syncthreads (global memory
// written by the CTA is visible to it after one).
constexpr int kAggregateOneCta = 4096, kAggregateOneCtaEntries = 65536;  // rows, entries

template <int kG>
__device__ void match_in_block(const Matching &m, int rounds) {
    const int lane = threadIdx.x & 31, nt = blockDim.x;
    const int nv = m.vs.size();
    for (int v = threadIdx.x; v < nv; v += nt) {
        m.mate[v] = -1;
        m.taken[v] = 0;
    }
    for (int r = threadIdx.x; r <= rounds; r += nt) m.counts[r] = 0;
    __syncthreads();
    for (int round = 0; round < rounds; ++round) {
        const int n = round ? *const_cast<volatile int32_t *>(m.counts + round) : nv;
        if (n == 0) break;
        for (int k0 = (threadIdx.x - lane) / kG; k0 < n; k0 += nt / kG) {
            const int k = k0 + lane / kG;
            const int v = k < n ? m.at(round, k) : -1;
            const int p = propose<kG>(m, v, lane % kG, round == 0);
            if (v >= 0 && lane % kG == 0) m.proposal[v] = p;
        }
        __syncthreads();
        for (int k0 = threadIdx.x - lane; k0 < n; k0 += nt)
            accept_one(m, round, k0 + lane < n ? m.at(round, k0 + lane) : -1);
        __syncthreads();
    }
}

template <int N, class In, class Out>
__device__ void scan_in_block(int n, const In &in, const Out &out) {
    using namespace scan_detail;
    Counts<N> carry{};
    for (int first = 0; first < n; first += kMidThreads * kItems)
        scan_tile<N, kMidThreads>(first, n, in, out, carry);
    __syncthreads();
}

template <int kG>
__global__ void __launch_bounds__(scan_detail::kMidThreads, 1) aggregate_one_cta(const __grid_constant__ AggregateState s) {
    match_in_block<kG>(s.rows, s.rounds);
    scan_in_block<1>(s.n + 1, s.to_pairs.f, s.to_pairs);
    match_in_block<kG>(s.pairs, s.rounds);
    scan_in_block<1>(s.n + 1, s.to_aggregates.f, s.to_aggregates);
    for (int round = 0; s.absorb && round < 2; ++round) {
        const int lane = threadIdx.x % kG, groups = blockDim.x / kG;
        for (int i = threadIdx.x / kG; i < s.n; i += groups) {
            if (proposes(s.absorption, i)) propose_absorption<kG>(s.absorption, i, lane);
            else if (lane == 0) s.absorption.proposal[i] = -1;
        }
        __syncthreads();
        for (int c = threadIdx.x / kG; c < s.n; c += groups)
            if (accepts(s.absorption, c)) accept_absorption<kG>(s.absorption, c, lane);
        __syncthreads();
    }
    scan_in_block<4>(s.n + 1, s.size_of, s.pack);
}

// Temporary arrays of a matching over at most n vertices.
struct MatchBuffers {
    Temp<int32_t> mate, proposal, open0, open1, counts;
    Temp<uint8_t> taken;
    MatchBuffers(tf_ctx *ctx, int n, int rounds)
        : mate(ctx, static_cast<size_t>(n)), proposal(ctx, static_cast<size_t>(n)),
          open0(ctx, static_cast<size_t>(n)), open1(ctx, static_cast<size_t>(n)),
          counts(ctx, static_cast<size_t>(rounds) + 1), taken(ctx, static_cast<size_t>(n)) {}
    Matching matching(const Vertices &vs, const Csr<double, int32_t> &g) const {
        return {vs, g.rp, g.ci, g.val, mate.data(), taken.data(), proposal.data(), {open0.data(), open1.data()},
                counts.data()};
    }
};

// Handshake rounds from an empty matching, two launches each.
void match_rounds(tf_ctx *ctx, const Matching &m, const Csr<double, int32_t> &g, int rounds) {
    memset_async(ctx, m.mate, 0xff, static_cast<size_t>(m.vs.n) * sizeof(int32_t));
    memset_async(ctx, m.taken, 0, static_cast<size_t>(m.vs.n));
    memset_async(ctx, m.counts, 0, (static_cast<size_t>(rounds) + 1) * sizeof(int32_t));
    // later rounds: an unknown, smaller number of vertices, in a grid stride
    const unsigned most = static_cast<unsigned>(ctx->sm_count) * 8;
    for (int r = 0; r < rounds; ++r) {
        with_row_lanes(g, [&](auto lanes) {
            constexpr int kG = decltype(lanes)::value;
            const unsigned grid = grid_for(static_cast<int64_t>(m.vs.n) * kG);
            match_propose<kG><<<r ? std::min(grid, most) : grid, kBlock, 0, ctx->stream>>>(m, r);
        });
        launched(ctx, "match_propose");
        const unsigned grid = grid_for(m.vs.n);
        match_accept<<<r ? std::min(grid, most) : grid, kBlock, 0, ctx->stream>>>(m, r);
        launched(ctx, "match_accept");
    }
}

}  // namespace

std::unique_ptr<tf_dcsr> canonicalize(tf_ctx *ctx, const Csr<double, int32_t> &a) {
    const int n = static_cast<int>(a.rows);
    Temp<uint64_t> keys(ctx, static_cast<size_t>(a.nnz));
    Temp<double> vals(ctx, static_cast<size_t>(a.nnz));
    const int bits = column_bits(n);
    map_entries<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, a.rp, a.ci, a.val, nullptr, keys.data(), vals.data(), bits);
    launched(ctx, "map_entries");
    return compress(ctx, n, a.nnz, keys.data(), vals.data(), bits, 0);
}

std::unique_ptr<tf_dcsr> strength_graph(tf_ctx *ctx, const Csr<double, int32_t> &a, const double *row_max,
                                        double theta) {
    require(std::isfinite(theta) && theta >= 0 && theta <= 1, "Invalid strength threshold");
    require(a.nnz <= INT32_MAX / 2, "Native AMG: strength graph exceeds 32-bit capacity", TF_ERR_LENGTH);
    const int n = static_cast<int>(a.rows);
    const int bits = column_bits(n);
    Temp<int32_t> count(ctx, static_cast<size_t>(n) + 1), offsets(ctx, static_cast<size_t>(n) + 1);
    memset_async(ctx, count.data() + n, 0, sizeof(int32_t));
    strength_edges<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, a.rp, a.ci, a.val, row_max, theta, nullptr, nullptr,
                                                            count.data(), bits);
    launched(ctx, "strength_count");
    scan_exclusive(ctx, n + 1, count.data(), offsets.data());
    const int32_t m = read_scalar(ctx, offsets.data() + n);
    Temp<uint64_t> keys(ctx, static_cast<size_t>(m));
    Temp<double> w(ctx, static_cast<size_t>(m));
    if (m) {
        strength_edges<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, a.rp, a.ci, a.val, row_max, theta, keys.data(),
                                                                w.data(), offsets.data(), bits);
        launched(ctx, "strength_fill");
    }
    return compress(ctx, n, m, keys.data(), w.data(), bits, 1);
}

template <class S, class V>
void level_arrays(tf_ctx *ctx, const Csr<double, int32_t> &a, const LevelArrays<S, V> &out, int *flags) {
    const int n = static_cast<int>(a.rows);
    with_row_lanes(a, [&](auto lanes) {
        constexpr int kG = decltype(lanes)::value;
        level_arrays_kernel<kG, S, V><<<grid_for(static_cast<int64_t>(n) * kG), kBlock, 0, ctx->stream>>>(
            n, a.rp, a.ci, a.val, out, flags);
    });
    launched(ctx, "level_arrays");
}
template void level_arrays<float, float>(tf_ctx *, const Csr<double, int32_t> &, const LevelArrays<float, float> &,
                                         int *);
template void level_arrays<double, double>(tf_ctx *, const Csr<double, int32_t> &, const LevelArrays<double, double> &,
                                           int *);
template void level_arrays<double, float>(tf_ctx *, const Csr<double, int32_t> &, const LevelArrays<double, float> &,
                                          int *);

void strength_weights(tf_ctx *ctx, const Csr<double, int32_t> &a, const double *row_max, double theta, double *w,
                      int *flags) {
    require(std::isfinite(theta) && theta >= 0 && theta <= 1, "Invalid strength threshold");
    require(a.nnz <= INT32_MAX / 2, "Native AMG: strength graph exceeds 32-bit capacity", TF_ERR_LENGTH);
    const int n = static_cast<int>(a.rows);
    memset_async(ctx, flags, 0, sizeof(int));
    with_row_lanes(a, [&](auto lanes) {
        constexpr int kG = decltype(lanes)::value;
        strength_weights_kernel<kG><<<grid_for(static_cast<int64_t>(n) * kG), kBlock, 0, ctx->stream>>>(
            n, a.rp, a.ci, a.val, row_max, theta, w, flags);
    });
    launched(ctx, "strength_weights");
}

int match_pairs(tf_ctx *ctx, const Csr<double, int32_t> &g, int rounds, int32_t *map) {
    require(rounds >= 1 && rounds <= 8, "Invalid matching configuration");
    const int n = static_cast<int>(g.rows);
    MatchBuffers buffers(ctx, n, rounds);
    Temp<int32_t> count(ctx, 1);
    Vertices vs;
    vs.n = n;
    const Matching m = buffers.matching(vs, g);
    match_rounds(ctx, m, g, rounds);
    const RootFlag root{vs, m.mate};
    scan_apply<1>(ctx, n + 1, root, AssignPairs{root, nullptr, nullptr, map, count.data()}, "assign_pairs");
    return read_scalar(ctx, count.data());
}

std::unique_ptr<tf_dcsr> contract_graph(tf_ctx *ctx, const Csr<double, int32_t> &g, const int32_t *map, int count) {
    const int n = static_cast<int>(g.rows);
    const int bits = column_bits(count);
    Temp<int32_t> cnt(ctx, static_cast<size_t>(n) + 1), offsets(ctx, static_cast<size_t>(n) + 1);
    memset_async(ctx, cnt.data() + n, 0, sizeof(int32_t));
    map_graph<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, g.rp, g.ci, g.val, map, cnt.data(), nullptr, nullptr, bits);
    launched(ctx, "map_graph_count");
    scan_exclusive(ctx, n + 1, cnt.data(), offsets.data());
    const int32_t m = read_scalar(ctx, offsets.data() + n);
    Temp<uint64_t> keys(ctx, static_cast<size_t>(m));
    Temp<double> vals(ctx, static_cast<size_t>(m));
    if (m) {
        map_graph<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, g.rp, g.ci, g.val, map, offsets.data(), keys.data(),
                                                           vals.data(), bits);
        launched(ctx, "map_graph_fill");
    }
    return compress(ctx, count, m, keys.data(), vals.data(), bits, 1);
}

// Two matchings (rows into pairs, pairs into aggregates), two absorption
// rounds and one compaction: the counts stay on the device until the end.
std::unique_ptr<tf_transfer> aggregate(tf_ctx *ctx, const Csr<double, int32_t> &g, int rounds, bool absorb,
                                       const int *strength_flags, int *flags) {
    require(rounds >= 1 && rounds <= 8 && g.rows > 0, "Invalid matching configuration");
    const int n = static_cast<int>(g.rows);
    const size_t sn = static_cast<size_t>(n);
    auto t = std::make_unique<tf_transfer>();
    t->fine_rows = n;
    t->map.allocate(sn);
    t->members.allocate(sn);
    int32_t *map = t->map.data();
    struct Result {
        int32_t pairs, aggregates, coarse, histogram[4], flags;
    };
    Temp<Result> result(ctx, 1);
    memset_async(ctx, result.data(), 0, sizeof(Result));
    Result *res = result.data();
    MatchBuffers buffers(ctx, n, rounds);
    Temp<int32_t> lo(ctx, sn), hi(ctx, sn), sizes(ctx, sn), slots(ctx, 4 * sn), off(ctx, sn + 1);
    Temp<double> scores(ctx, absorb ? sn : 0);
    Vertices rows, pairs;
    rows.n = n;
    pairs.lo = lo.data();
    pairs.hi = hi.data();
    pairs.map = map;
    pairs.count = &res->pairs;
    pairs.n = n;
    AggregateState s;
    s.n = n;
    s.rounds = rounds;
    s.absorb = absorb;
    s.rows = buffers.matching(rows, g);
    s.pairs = buffers.matching(pairs, g);
    s.to_pairs = {{rows, s.rows.mate}, lo.data(), hi.data(), map, &res->pairs};
    s.to_aggregates = {{pairs, s.pairs.mate}, slots.data(), sizes.data(), map, &res->aggregates};
    s.absorption = {g.rp, g.ci, g.val, &res->aggregates, map, sizes.data(), slots.data(), s.rows.proposal,
                    scores.data()};
    s.size_of = {sizes.data(), &res->aggregates};
    s.pack = {n, slots.data(), off.data(), t->members.data(), map, &res->coarse, res->histogram, strength_flags,
              &res->flags};
    if (n <= kAggregateOneCta && g.nnz <= kAggregateOneCtaEntries) {
        with_row_lanes(g, [&](auto lanes) {
            aggregate_one_cta<decltype(lanes)::value><<<1, scan_detail::kMidThreads, 0, ctx->stream>>>(s);
        });
        launched(ctx, "aggregate_one_cta");
    } else {
        match_rounds(ctx, s.rows, g, rounds);
        scan_apply<1>(ctx, n + 1, s.to_pairs.f, s.to_pairs, "assign_pairs");
        match_rounds(ctx, s.pairs, g, rounds);
        scan_apply<1>(ctx, n + 1, s.to_aggregates.f, s.to_aggregates, "assign_aggregates");
        for (int round = 0; absorb && round < 2; ++round) {
            with_row_lanes(g, [&](auto lanes) {
                constexpr int kG = decltype(lanes)::value;
                const unsigned lanes_grid = grid_for(static_cast<int64_t>(n) * kG);
                propose_absorption_kernel<kG>
                    <<<kG == 32 ? lanes_grid : grid_for(n), kBlock, 0, ctx->stream>>>(n, s.absorption);
                launched(ctx, "propose_absorption");
                accept_absorption_kernel<kG><<<lanes_grid, kBlock, 0, ctx->stream>>>(n, s.absorption);
                launched(ctx, "accept_absorption");
            });
        }
        scan_apply<4>(ctx, n + 1, s.size_of, s.pack, "pack_aggregates");
    }
    const Result r = read_scalar(ctx, res);
    if (flags) *flags = r.flags;
    t->coarse_rows = r.coarse;
    for (int k = 0; k < 4; ++k) t->histogram[k] = r.histogram[k];
    t->offsets.allocate(static_cast<size_t>(r.coarse) + 1);
    copy_async(ctx, t->offsets.data(), off.data(), (static_cast<size_t>(r.coarse) + 1) * sizeof(int32_t));
    cuda_check(cudaStreamSynchronize(ctx->stream), "aggregate");
    return t;
}

std::unique_ptr<tf_dcsr> galerkin(tf_ctx *ctx, const Csr<double, int32_t> &a, const int32_t *map, int coarse) {
    const int n = static_cast<int>(a.rows);
    require(coarse >= 1, "AMG transfer dimension mismatch");
    const int bits = column_bits(coarse);
    Temp<uint64_t> keys(ctx, static_cast<size_t>(a.nnz));
    Temp<double> vals(ctx, static_cast<size_t>(a.nnz));
    map_entries<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, a.rp, a.ci, a.val, map, keys.data(), vals.data(), bits);
    launched(ctx, "map_entries");
    return compress(ctx, coarse, a.nnz, keys.data(), vals.data(), bits, 0);
}

std::unique_ptr<tf_dcsr> galerkin(tf_ctx *ctx, const Csr<double, int32_t> &a, const tf_transfer &t) {
    const int coarse = t.coarse_rows;
    require(coarse >= 1, "AMG transfer dimension mismatch");
    const int32_t *off = t.offsets.data(), *mem = t.members.data(), *map = t.map.data();
    Temp<int32_t> base(ctx, static_cast<size_t>(coarse) + 1), count(ctx, static_cast<size_t>(coarse) + 1);
    int *longest = static_cast<int *>(ctx->arena(sizeof(int), 1));
    memset_async(ctx, longest, 0, sizeof(int));
    merged_lengths<<<grid_for(coarse + 1), kBlock, 0, ctx->stream>>>(coarse, off, mem, a.rp, count.data(), longest);
    launched(ctx, "merged_lengths");
    scan_exclusive(ctx, coarse + 1, count.data(), base.data());
    const int most = read_scalar(ctx, longest);
    if (most > kMergeMax) return galerkin(ctx, a, map, coarse);
    Temp<int32_t> tcol(ctx, static_cast<size_t>(a.nnz));
    Temp<double> tval(ctx, static_cast<size_t>(a.nnz));
    auto merge = [&](auto kmax, auto warps) {
        constexpr int kMax = decltype(kmax)::value, kWarps = decltype(warps)::value;
        auto go = [&](auto kernel) {
            kernel<<<grid_for(coarse + 1, kWarps), kWarps * 32, 0, ctx->stream>>>(coarse, off, mem, a.rp, a.ci, a.val,
                                                                                  map, base.data(), tcol.data(),
                                                                                  tval.data(), count.data());
        };
        // (31 bits: no key equals the padding key)
        if (column_bits(coarse) + merge_seq_bits(kMax) <= 31) go(merge_rows<kMax, kWarps, uint32_t>);
        else go(merge_rows<kMax, kWarps, uint64_t>);
        launched(ctx, "merge_rows");
    };
    using std::integral_constant;
    if (most <= 32) merge(integral_constant<int, 1>{}, integral_constant<int, 8>{});
    else if (most <= 64) merge(integral_constant<int, 2>{}, integral_constant<int, 8>{});
    else if (most <= 128) merge(integral_constant<int, 4>{}, integral_constant<int, 8>{});
    else if (most <= 256) merge(integral_constant<int, 8>{}, integral_constant<int, 8>{});
    else merge(integral_constant<int, 16>{}, integral_constant<int, 4>{});
    auto out = std::make_unique<tf_dcsr>();
    out->rows = out->cols = coarse;
    out->offsets.allocate(static_cast<size_t>(coarse + 1) * sizeof(int32_t));
    auto *rp = reinterpret_cast<int32_t *>(out->offsets.data());
    scan_exclusive(ctx, coarse + 1, count.data(), rp);
    out->nnz = read_scalar(ctx, rp + coarse);
    out->indices.allocate(static_cast<size_t>(out->nnz) * sizeof(int32_t));
    out->values.allocate(static_cast<size_t>(out->nnz) * sizeof(double));
    if (out->nnz) {
        pack_rows<<<grid_for(static_cast<int64_t>(coarse) * 8), kBlock, 0, ctx->stream>>>(
            coarse, base.data(), rp, tcol.data(), tval.data(), reinterpret_cast<int32_t *>(out->indices.data()),
            reinterpret_cast<double *>(out->values.data()));
        launched(ctx, "pack_rows");
    }
    return out;
}

}  // namespace tfb
