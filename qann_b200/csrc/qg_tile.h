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
void tile_prepare_queries(const float* rows, size_t n, int dim, TileQueries& out, cudaStream_t st);
void tile_prepare_base(const float* rows, size_t n, int dim, TileBase& out, cudaStream_t st);

// Each query's nearest base row by squared L2 (the smallest score, the first
// row on ties; exact: see qg_tile.cu) in label[nq]. Queries the engine could
// not settle are listed in redo (their count returned): the caller redoes
// those exactly. q, base_rows: the float rows behind qs and base.
size_t tile_nearest(const float* q, const TileQueries& qs, const float* base_rows, const TileBase& base,
                    uint32_t* label, DevBuf<uint32_t>& redo, cudaStream_t st);

// The epilogue-warp autotuner: on or off, problems tuned, the last launch's pick.
// force: 0 the autotuner's pick; 8 or 16 that epilogue on every launch.
void set_tile_autotune(int on);
int tile_autotune();
int64_t tile_tuned_problems();
int tile_last_epilogue_warps();
void set_tile_epilogue_warps(int warps);
int tile_epilogue_warps();

} // namespace qg
