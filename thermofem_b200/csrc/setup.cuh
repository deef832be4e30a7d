// setup.cuh -- typed entry points of the sorting primitives (sort.cu) and of
// the aggregation setup's stages (setup.cu).
#pragma once
#include "ops.cuh"

namespace tfb {

// Sorting primitives (sort.cu).
void radix_sort_pairs(tf_ctx *ctx, int64_t n, const uint64_t *kin, const double *vin, uint64_t *kout,
                      double *vout, int end_bit);
int64_t reduce_by_key(tf_ctx *ctx, int64_t n, const uint64_t *keys, const double *vals, int op, uint64_t *kout,
                      double *vout);

// Coordinate compression (sort + reduce + unpack) into an owned CSR.
std::unique_ptr<tf_dcsr> compress(tf_ctx *ctx, int rows, int64_t n, const uint64_t *keys, const double *vals, int col_bits, int op);
int column_bits(int rows);

// Setup stages (setup.cu), on canonical FP64/int32 operands.
std::unique_ptr<tf_dcsr> canonicalize(tf_ctx *ctx, const Csr<double, int32_t> &a);
std::unique_ptr<tf_dcsr> strength_graph(tf_ctx *ctx, const Csr<double, int32_t> &a, const double *row_max, double theta);
int match_pairs(tf_ctx *ctx, const Csr<double, int32_t> &g, int rounds, int32_t *map);
std::unique_ptr<tf_dcsr> contract_graph(tf_ctx *ctx, const Csr<double, int32_t> &g, const int32_t *map, int count);
// Where a level's arrays go: structure, stored values, inverse diagonal,
// columns as row offsets (null: none wanted), largest |off-diagonal| per row.
template <class S, class V>
struct LevelArrays {
    int32_t *rp, *ci;
    V *val;
    S *dinv;
    int16_t *cd;
    double *row_max;
};
// Flags (device, zeroed by the caller): a value, diagonal or its reciprocal is
// not usable (row_stats); the diagonal does not invert in S; a column lies
// further than 32,767 from its row.
constexpr int kLevelInvalid = 1, kLevelDiagonal = 2, kLevelWide = 4;
template <class S, class V>
void level_arrays(tf_ctx *ctx, const Csr<double, int32_t> &a, const LevelArrays<S, V> &out, int *flags);

// The strength graph on a's own pattern: w[j] the weight of entry j's edge,
// 0 where it is weak.  *flags (device): bit 0 some edge is strong; bit 1 a
// strong edge has no entry for its other direction, and strength_graph has to
// be taken instead.
constexpr int kStrengthSome = 1, kStrengthUnsymmetric = 2;
void strength_weights(tf_ctx *ctx, const Csr<double, int32_t> &a, const double *row_max, double theta, double *w,
                      int *flags);
// Edges of weight 0 are none.  strength_flags (device) and flags: the former's
// value, read back with the results.
std::unique_ptr<tf_transfer> aggregate(tf_ctx *ctx, const Csr<double, int32_t> &g, int rounds, bool absorb,
                                       const int *strength_flags = nullptr, int *flags = nullptr);
// P^T A P for any map, by a sort over all coordinates, and for a transfer's
// aggregates (at most four members), row by row; the same bits.
std::unique_ptr<tf_dcsr> galerkin(tf_ctx *ctx, const Csr<double, int32_t> &a, const int32_t *map, int coarse);
std::unique_ptr<tf_dcsr> galerkin(tf_ctx *ctx, const Csr<double, int32_t> &a, const tf_transfer &t);

}  // namespace tfb
