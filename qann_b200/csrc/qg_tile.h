// The tensor-core tile engine: products of query rows with base rows in F16,
// read out as raw products, as lower bounds below a threshold, or as each
// query's nearest row (qg_tile.cu).
#pragma once

#include "qg_cuda.h"

#include <cstddef>
#include <cstdint>

namespace qg {

// Query rows for the engine: each row scaled by its own power of two (2^exps)
// and rounded to f16, zero-padded to dpad (a multiple of 8), with the float
// squared norms of the unscaled rows.
struct TileQueries {
    size_t n = 0;
    int dim = 0, dpad = 0;
    DevBuf<uint16_t> f16;
    DevBuf<float> sq;
    DevBuf<int> exps;
};

// Base rows for the engine: one power of two for every row, taken from the
// largest magnitude among them (amax, its bits), the rest as above. Rows whose
// squared norm is extreme (tile_extreme) are zero in f16.
struct TileBase {
    size_t n = 0;
    int dim = 0, dpad = 0;
    DevBuf<uint16_t> f16;
    DevBuf<float> sq;
    DevBuf<uint32_t> amax;
};

// Dimensions the engine takes.
bool tile_supported(int dim);
// The device memory of n prepared query rows.
inline size_t tile_query_bytes(size_t n, int dim) {
    return n * ((static_cast<size_t>(dim) + 7) / 8 * 8 * sizeof(uint16_t) + sizeof(float) + sizeof(int));
}
void tile_prepare_queries(const float* rows, size_t n, int dim, TileQueries& out, cudaStream_t st);
// The device memory of n prepared base rows.
inline size_t tile_base_bytes(size_t n, int dim) {
    return n * ((static_cast<size_t>(dim) + 7) / 8 * 8 * sizeof(uint16_t) + sizeof(float));
}
void tile_prepare_base(const float* rows, size_t n, int dim, TileBase& out, cudaStream_t st);

// Each query's nearest base row by squared L2 (the smallest score, the first
// row on ties; exact: see qg_tile.cu) in label[nq]. Queries the engine could
// not settle are listed in redo (their count returned): the caller redoes
// those exactly. q, base_rows: the float rows behind qs and base.
size_t tile_nearest(const float* q, const TileQueries& qs, const float* base_rows, const TileBase& base,
                    uint32_t* label, DevBuf<uint32_t>& redo, cudaStream_t st);

// The exact k nearest base rows of each query by (score, row), -0 == +0:
// out_key[nq][k] (key_eq0(score) << 32 | row, ~0 when there are fewer) and
// out_slot[nq][k], sorted. ip: the score is -(q . x), else squared L2. allow /
// deny: bitmaps over the rows, or null. k at most kTileMaxK. Queries not settled are
// listed in redo[0 .. nq): from its start those that the sweep form settles as a rule
// (rows stored in an order), at its end those that want the exact path.
inline constexpr size_t kTileMaxK = 1024;
struct TileRedo {
    size_t sweep = 0, exact = 0;   // redo[0 .. sweep) and redo[nq - exact .. nq)
};
TileRedo tile_topk(const float* q, const TileQueries& qs, const float* base_rows, const TileBase& base, bool ip, size_t k,
                   const uint64_t* allow, const uint64_t* deny, uint64_t* out_key, uint32_t* out_slot,
                   DevBuf<uint32_t>& redo, bool sweep, cudaStream_t st);

// The raw products of the queries with n base rows (f16 rows of dpad
// elements), row after row of `store` (ld apart). *err is set if a pipeline
// wait times out; with may_tune false nothing waits on the host.
void tile_store(const TileQueries& qs, const uint16_t* base_f16, size_t n, int dpad, float* store, size_t ld, int* err,
                bool may_tune, cudaStream_t st);

// C of the error bound (qg_tile.cu).
double tile_error_factor(int dim);

// The epilogue-warp autotuner: on or off, problems tuned, the last launch's pick.
// force: 0 the autotuner's pick; 8 or 16 that epilogue on every launch.
void set_tile_autotune(int on);
int tile_autotune();
int64_t tile_tuned_problems();
int tile_last_epilogue_warps();
void set_tile_epilogue_warps(int warps);
int tile_epilogue_warps();

} // namespace qg
