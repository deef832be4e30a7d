// setup.cu -- device stages of the aggregation AMG setup: canonical form,
// strength graph, synchronous handshake matching, graph contraction,
// singleton absorption, member tables and the Galerkin product.
//
// The algorithm is the reference's (src/Multigrid/GpuAggregation.cu, whose
// host statement is test/support/NativeAggregationOracle.cu); the results
// (aggregates, member order, histograms, coarse sparsity) are meant to be
// bit-identical to it, which is why every stage keeps the reference's
// snapshot semantics: proposals of a matching round are all written before
// any are accepted, absorption reads the pre-round map and sizes, member
// slots are re-sorted after the atomic fill.  Sorting, reduction and scans
// are the project's own (sort.cu).
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

// State of a matching between rounds: mate[] (-1 unmatched) as of the
// proposals before last, and the last round's proposals, not yet accepted:
// a mutual pair among them is matched.  Vertex v's own thread writes that
// into mate[v] in the next round; readers that still find -1 there come to
// the same answer from the proposals.
__device__ __forceinline__ int mate_of(int v, const int32_t *mate, const int32_t *last) {
    const int m = mate[v];
    if (m >= 0 || !last) return m;
    const int p = last[v];
    return p >= 0 && last[p] == v ? p : -1;
}

// (s, c) beats (score, best) as v's proposal (GpuAggregation.cu:402-431):
// larger weight, then larger edge priority, then smaller vertex.
__device__ __forceinline__ bool better(int v, double s, int c, double score, int best) {
    if (s != score) return s > score;
    if (c < 0 || c == best) return false;
    if (best < 0) return s > 0;
    const uint64_t a = edge_priority(v, c), b = edge_priority(v, best);
    return a > b || (a == b && c < best);
}

// One handshake round: accepts the last round's mutual proposals
// (GpuAggregation.cu:440-449) and writes this round's: each unmatched vertex
// proposes its best unmatched neighbour, from one snapshot of the matching.
// kG lanes share a vertex.
//
// Bound: the gathers of the neighbours' state.  Acceptance in the next
// round's kernel halves the launches of a matching; weights are read first,
// and only an edge that would win gathers its neighbour.
template <int kG>
__global__ void match_round(Vertices vs, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                            const double *__restrict__ w, int32_t *mate, const int32_t *__restrict__ last,
                            int32_t *__restrict__ proposal) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int lane = static_cast<int>(t % kG);
    const int nv = vs.size();
    if (t / kG >= nv) return;  // uniform over the vertex's lanes
    const int v = static_cast<int>(t / kG);
    const int mine = mate_of(v, mate, last);
    if (mine >= 0) {
        if (lane == 0) {
            mate[v] = mine;
            proposal[v] = -1;
        }
        return;
    }
    int best = -1;
    double score = 0;
    for (int k = 0; k < 2; ++k) {
        const int row = vs.lo ? (k ? vs.hi[v] : vs.lo[v]) : (k ? -1 : v);
        if (row < 0) break;
        for (int32_t j = rp[row] + lane; j < rp[row + 1]; j += kG) {
            const double s = w[j];
            if (!(s > 0) || s < score) continue;
            const int c = vs.of(ci[j]);
            if (c == v || !better(v, s, c, score, best) || mate_of(c, mate, last) >= 0) continue;
            best = c;
            score = s;
        }
    }
    if constexpr (kG > 1) {
        const unsigned group = (kG == 32 ? 0xffffffffu : ((1u << (kG & 31)) - 1u))
                               << ((threadIdx.x & 31) / kG * kG);
#pragma unroll
        for (int o = kG / 2; o > 0; o >>= 1) {
            const double s = __shfl_xor_sync(group, score, o);
            const int c = __shfl_xor_sync(group, best, o);
            if (better(v, s, c, score, best)) {
                best = c;
                score = s;
            }
        }
    }
    if (lane == 0) proposal[v] = best;
}

// Scan input: 1 for the vertex that stands for its pair (or itself alone).
struct RootFlag {
    Vertices vs;
    const int32_t *mate, *last;
    __device__ Counts<1> operator()(int v) const {
        if (v >= vs.size()) return {0};
        const int m = mate_of(v, mate, last);
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
        const int m = mate_of(v, f.mate, f.last);
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
        const int m = mate_of(v, f.mate, f.last);
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
__global__ void propose_absorption(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                   const double *__restrict__ w, const int32_t *__restrict__ map,
                                   const int32_t *__restrict__ sizes, int32_t *__restrict__ proposal,
                                   double *__restrict__ scores) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int best = -1;
    double score = 0;
    if (sizes[map[i]] == 1) {
        for (int32_t j = rp[i]; j < rp[i + 1]; ++j) {
            const int c = map[ci[j]];
            const double s = w[j];
            if (sizes[c] < 2 || sizes[c] >= 4 || s <= 0) continue;
            if (s > score || (s == score && (best < 0 || c < best))) {
                best = c;
                score = s;
            }
        }
    }
    proposal[i] = best;
    scores[i] = score;
}

// Each target keeps its best distinct proposers, weight descending then
// fine id ascending, up to its remaining capacity (GpuAggregation.cu:685-720),
// and takes them in: map, slots and sizes are updated in place.  A thread
// reads only its own aggregate's size and slots (a singleton's size may turn
// from 1 to 0 under its own thread, which has nothing to do either way), and
// the proposals of the kernel before.
__global__ void accept_absorption(const int32_t *count, const int32_t *__restrict__ rp,
                                  const int32_t *__restrict__ ci, int32_t *sizes, int32_t *slots,
                                  const int32_t *__restrict__ proposal, const double *__restrict__ scores,
                                  int32_t *map) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= *count) return;
    const int size = sizes[c];
    if (size < 2 || size >= 4) return;
    int sel[2] = {-1, -1};
    double sw[2] = {-1, -1};
    const int cap = 4 - size;
    for (int k = 0; k < size; ++k) {
        const int row = slots[static_cast<int64_t>(c) * 4 + k];
        for (int32_t j = rp[row]; j < rp[row + 1]; ++j) {
            const int i = ci[j];
            if (proposal[i] != c || i == sel[0] || i == sel[1]) continue;
            const double s = scores[i];
            for (int q = 0; q < cap; ++q) {
                if (s > sw[q] || (s == sw[q] && i < sel[q])) {
                    for (int r = cap - 1; r > q; --r) {
                        sel[r] = sel[r - 1];
                        sw[r] = sw[r - 1];
                    }
                    sel[q] = i;
                    sw[q] = s;
                    break;
                }
            }
        }
    }
    int now = size;
    for (int q = 0; q < cap; ++q) {
        if (sel[q] < 0) continue;
        sizes[map[sel[q]]] = 0;
        map[sel[q]] = c;
        slots[static_cast<int64_t>(c) * 4 + now++] = sel[q];
    }
    if (now != size) sizes[c] = now;
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
template <int K>
__device__ __forceinline__ void warp_sort(uint64_t (&k)[K], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= K) {
                const int lx = stride / K;
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    const uint64_t other = __shfl_xor_sync(0xffffffffu, k[r], lx);
                    const bool up = ((lane * K + r) & size) == 0, lower = (lane & lx) == 0;
                    k[r] = (up == lower) == (k[r] < other) ? k[r] : other;
                }
            } else {
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    if (r & stride) continue;
                    const bool up = ((lane * K + r) & size) == 0;
                    const uint64_t a = k[r], b = k[r | stride];
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

// Row c of P^T A P (one warp): its members' entries (col = map[ci], in member
// and entry order) sorted by (column, that order); each run of a column is
// then added left to right, the order in which the stable sort over all
// coordinates adds it, so the sums are the same bits.  The row goes to
// tcol/tval from base[c], its length to count[c].
//
// Bound: instructions, not memory.  128^3 finest level (598k rows of 24
// entries): 0.19 ms against 3.4 ms for map, sort, reduce and unpack.  K keys
// per lane is the smallest power of two that holds the level's longest row.
template <int K, int kWarps>
__global__ void __launch_bounds__(kWarps * 32) merge_rows(int coarse, const int32_t *__restrict__ off,
                                                          const int32_t *__restrict__ mem,
                                                          const int32_t *__restrict__ rp,
                                                          const int32_t *__restrict__ ci,
                                                          const double *__restrict__ a,
                                                          const int32_t *__restrict__ map,
                                                          const int32_t *__restrict__ base, int32_t *__restrict__ tcol,
                                                          double *__restrict__ tval, int32_t *__restrict__ count) {
    constexpr int kCap = 32 * K;
    __shared__ double s_val[kWarps][kCap];
    __shared__ int32_t s_col[kWarps][kCap];
    __shared__ uint16_t s_seq[kWarps][kCap];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * kWarps + warp;
    if (c >= coarse) {
        if (c == coarse && lane == 0) count[c] = 0;  // the scan's sentinel
        return;
    }
    double *val = s_val[warp];
    int32_t *col = s_col[warp];
    uint16_t *seq = s_seq[warp];
    const int o0 = off[c], members = off[c + 1] - o0;
    int start = 0, len = 0;
    if (lane < members) {
        const int m = mem[o0 + lane];
        start = rp[m];
        len = rp[m + 1] - start;
    }
    const int p1 = __shfl_sync(0xffffffffu, len, 0), p2 = p1 + __shfl_sync(0xffffffffu, len, 1),
              p3 = p2 + __shfl_sync(0xffffffffu, len, 2), n = p3 + __shfl_sync(0xffffffffu, len, 3);
    // entry q of the merged list is entry q + shift of A within its member
    const int s0 = __shfl_sync(0xffffffffu, start, 0), s1 = __shfl_sync(0xffffffffu, start, 1) - p1,
              s2 = __shfl_sync(0xffffffffu, start, 2) - p2, s3 = __shfl_sync(0xffffffffu, start, 3) - p3;
    uint64_t key[K];
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const int q = r * 32 + lane;
        key[r] = ~uint64_t(0);
        if (q < n) {
            const int j = q + (q < p1 ? s0 : (q < p2 ? s1 : (q < p3 ? s2 : s3)));
            key[r] = (static_cast<uint64_t>(static_cast<unsigned>(map[ci[j]])) << 16) | static_cast<unsigned>(q);
            val[q] = a[j];
        }
    }
    warp_sort<K>(key, lane);
    const uint64_t before = __shfl_up_sync(0xffffffffu, key[K - 1], 1);
    unsigned heads = 0;
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const int e = lane * K + r;
        if (e < n) {
            const int32_t mine = static_cast<int32_t>(key[r] >> 16);
            col[e] = mine;
            seq[e] = static_cast<uint16_t>(key[r] & 0xffffu);
            const uint64_t left = r > 0 ? key[r > 0 ? r - 1 : 0] : before;
            if (e == 0 || static_cast<int32_t>(left >> 16) != mine) heads |= 1u << r;
        }
    }
    __syncwarp();
    int inc = __popc(heads);
    const int own = inc;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) count[c] = inc;
    int out = base[c] + inc - own;
#pragma unroll
    for (int r = 0; r < K; ++r) {
        if (!(heads >> r & 1u)) continue;
        const int e = lane * K + r;
        const int32_t mine = col[e];
        double sum = val[seq[e]];
        for (int q = e + 1; q < n && col[q] == mine; ++q) sum += val[seq[q]];
        tcol[out] = mine;
        tval[out] = sum;
        ++out;
    }
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

// Handshake rounds over vs from an empty matching; the state after them is
// (mate, *last).
void match_rounds(tf_ctx *ctx, const Vertices &vs, const Csr<double, int32_t> &g, int rounds, int32_t *mate,
                  int32_t *prop0, int32_t *prop1, const int32_t **last) {
    memset_async(ctx, mate, 0xff, static_cast<size_t>(vs.n) * sizeof(int32_t));
    *last = nullptr;
    for (int r = 0; r < rounds; ++r) {
        int32_t *proposal = r & 1 ? prop1 : prop0;
        with_row_lanes(g, [&](auto lanes) {
            constexpr int kG = decltype(lanes)::value;
            match_round<kG><<<grid_for(static_cast<int64_t>(vs.n) * kG), kBlock, 0, ctx->stream>>>(
                vs, g.rp, g.ci, g.val, mate, *last, proposal);
        });
        launched(ctx, "match_round");
        *last = proposal;
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
    Temp<int32_t> mate(ctx, static_cast<size_t>(n)), prop0(ctx, static_cast<size_t>(n)),
        prop1(ctx, static_cast<size_t>(n)), count(ctx, 1);
    Vertices vs;
    vs.n = n;
    const int32_t *last = nullptr;
    match_rounds(ctx, vs, g, rounds, mate.data(), prop0.data(), prop1.data(), &last);
    const RootFlag root{vs, mate.data(), last};
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
// rounds, and one compaction, in one stretch of launches: the counts stay on
// the device until the end.
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
    Temp<int32_t> mate(ctx, sn), prop0(ctx, sn), prop1(ctx, sn), lo(ctx, sn), hi(ctx, sn), sizes(ctx, sn),
        slots(ctx, 4 * sn), off(ctx, sn + 1);
    const int32_t *last = nullptr;
    Vertices rows;
    rows.n = n;
    match_rounds(ctx, rows, g, rounds, mate.data(), prop0.data(), prop1.data(), &last);
    const RootFlag row_root{rows, mate.data(), last};
    scan_apply<1>(ctx, n + 1, row_root, AssignPairs{row_root, lo.data(), hi.data(), map, &res->pairs}, "assign_pairs");
    Vertices pairs;
    pairs.lo = lo.data();
    pairs.hi = hi.data();
    pairs.map = map;
    pairs.count = &res->pairs;
    pairs.n = n;
    match_rounds(ctx, pairs, g, rounds, mate.data(), prop0.data(), prop1.data(), &last);
    const RootFlag pair_root{pairs, mate.data(), last};
    scan_apply<1>(ctx, n + 1, pair_root,
                  AssignAggregates{pair_root, slots.data(), sizes.data(), map, &res->aggregates}, "assign_aggregates");
    if (absorb) {
        Temp<double> scores(ctx, sn);
        int32_t *proposal = prop0.data();
        for (int round = 0; round < 2; ++round) {
            propose_absorption<<<grid_for(n), kBlock, 0, ctx->stream>>>(n, g.rp, g.ci, g.val, map, sizes.data(),
                                                                        proposal, scores.data());
            launched(ctx, "propose_absorption");
            accept_absorption<<<grid_for(n), kBlock, 0, ctx->stream>>>(&res->aggregates, g.rp, g.ci, sizes.data(),
                                                                       slots.data(), proposal, scores.data(), map);
            launched(ctx, "accept_absorption");
        }
    }
    scan_apply<4>(ctx, n + 1, SizeOf{sizes.data(), &res->aggregates},
                  PackAggregates{n, slots.data(), off.data(), t->members.data(), map, &res->coarse, res->histogram,
                                 strength_flags, &res->flags},
                  "pack_aggregates");
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
    auto merge = [&](auto kernel, int warps) {
        kernel<<<grid_for(coarse + 1, warps), warps * 32, 0, ctx->stream>>>(coarse, off, mem, a.rp, a.ci, a.val, map,
                                                                            base.data(), tcol.data(), tval.data(),
                                                                            count.data());
        launched(ctx, "merge_rows");
    };
    if (most <= 32) merge(merge_rows<1, 8>, 8);
    else if (most <= 64) merge(merge_rows<2, 8>, 8);
    else if (most <= 128) merge(merge_rows<4, 8>, 8);
    else if (most <= 256) merge(merge_rows<8, 8>, 8);
    else merge(merge_rows<16, 4>, 4);
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
