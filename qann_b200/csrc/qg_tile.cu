// The tensor-core tile engine. One persistent, warp-specialised kernel forms
// acc(q, x) = dot of f16 query and base rows, accumulated in FP32 in TMEM, in
// tiles of 256 queries by 128 base rows, and its epilogue reads them out by
// mode.
//
// Why results taken from it are exact. Query row q is scaled by 2^qe, the
// base rows by one 2^xe, so that the largest element lies in [2^13, 2^14), and
// rounded to f16 (unit roundoff u = 2^-11; below 2^-14 the spacing is 2^-24).
// With s the exact score as the reference computes it (squared L2, or -dot, in
// float, AVX2 order) and s^ = |q|^2 + |x|^2 - 2 acc 2^-(qe+xe) (or -acc
// 2^-(qe+xe)) its estimate,
//   |s^ - s| <= e = c (|q|^2 + |x|^2) + g
//   c = C for L2, C / 2 for inner product; C = 2^-10 + 2^-13 + d 2^-21
//   g = 2 a for L2, a for inner product; a = sqrt(d) |q| M 2^-37
// (2u + u^2) sum|q_i x_i| comes from the relative rounding of both inputs and
// sum|q_i x_i| <= (|q|^2 + |x|^2) / 2; d 2^-21 covers the tensor cores' FP32
// accumulation; the 2^-13 the float rounding of the norms, of the bounds and
// of the reference's own score; a the absolute rounding of elements of a base
// row that are below 2^-27 of M, the largest magnitude in the base. Squared
// norms below 2^-100 or not below 2^100 (tile_extreme), where float squares
// lose relative accuracy, are left out of this: such a query is not settled
// here, and such a row always passes.
//
// Bounds are compared without the query's own terms, which are the same for
// all rows: lb = xterm(x) - mult acc 2^-(qe+xe) with xterm = (1 - C) |x|^2
// and mult = 2 for L2, xterm = -C / 2 |x|^2 and mult = 1 for inner product;
// the upper bound on the same scale is lb + 2 c |x|^2 + (2 c |q|^2 + 2 g).
#include "qg_device.cuh"
#include "qg_ops.h"
#include "qg_sm100.cuh"
#include "qg_tile.h"

#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>

namespace qg {

namespace {

constexpr int BM = 256;         // queries per tile: two halves of 128 TMEM lanes
constexpr int BN = 128;         // base rows per tile (accumulator columns of a half)
constexpr int KA = 64;          // f16 elements per 128-byte swizzle row (a K block)
constexpr int kMaxDim = 2048;
constexpr uint32_t kABlock = BM * 128, kBBlock = BN * 128;   // bytes of one K block
constexpr uint32_t kPipeBytes = 192 * 1024;                  // query buffers and the ring
constexpr int kSlots = 7;       // candidates a lane holds before it appends them
constexpr uint32_t kTmemCols = 512;   // two accumulators of two halves
constexpr float kOpen = 3.402823466e+38f;   // threshold of a query that has none yet
constexpr int kNearestCap = 256;            // candidates of a query in nearest mode
constexpr size_t kMaxChunkRows = size_t{1} << 22;   // base rows a launch
constexpr int kSweeps = 6;      // each leaves about cap / k times fewer rows that pass
constexpr int kMaxCap = 8192;   // candidates of a query in filter mode at most; lists are counted up to it
constexpr uint32_t kGivenUp = 0x80000000u;   // the count of a list that a sweep would not settle either

// What the epilogue does with an accumulator.
enum TileMode {
    kNearest,   // append rows below the running upper bound of each query's nearest
    kFilter,    // append rows below each query's threshold
    kStore,     // write the products
};

struct TileArgs {
    int nq;
    int n0;              // first base row of this launch, a multiple of 128; ntiles tiles from there
    int kblocks;         // 64-element K blocks of the padded rows
    int ksteps;          // 16-element MMA steps covering d
    int mtiles, ntiles, group_n;
    int ctas;            // at most so many CTAs, or 0
    int scout;           // nearest: tiles of each group first read for their bounds alone
    const float* xterm;      // per base row: its part of the lower bound (+inf: not to be returned), padded
                             // with +inf to whole tiles
    const float* run_slack;  // per 32 base rows: 2 c max|x|^2 (+inf when one of them is extreme), padded alike
    const float* qmul;       // per query: mult 2^-(qe+xe)
    const float* qslack;     // per query: 2 c |q|^2 + 2 g
    uint32_t* thr_key;       // per query: key of its threshold (nearest: the smallest upper bound so far)
    uint32_t* cand_count;    // per query
    uint2* cand;             // per query, cap entries: (lower bound, row)
    int cap;
    int* err;
    float* store;            // kStore: acc(q, row) at store[q * ld + row - n0], ncols columns
    size_t ld;
    int ncols;
};

// Where the pipeline's parts lie in shared memory. Up to two K blocks (d <=
// 128) the query tile is resident, double buffered when there are several, and
// the ring stages one K block of base rows; deeper rows stream both operands
// through the ring. (A batch of one query tile is bound by the base rows'
// stream from HBM and has the whole ring for them.)
struct TilePipe {
    bool resident;
    uint32_t a_bytes, stage_bytes, ring_at;
    int stages;
    __host__ __device__ TilePipe(int kblocks, int mtiles)
        : resident(kblocks <= 2),
          a_bytes(resident ? kblocks * kABlock : 0),
          stage_bytes(resident ? kBBlock : kABlock + kBBlock),
          ring_at(mtiles > 1 ? 2 * a_bytes : a_bytes),
          stages(static_cast<int>((kPipeBytes - ring_at) / stage_bytes)) {}
};
constexpr int kMaxStages = 10;
constexpr int kTermBufs = 8;                          // tiles whose row terms are staged ahead
constexpr uint32_t kTermBytes = BN * 4, kSlackBytes = BN / 32 * 4;
constexpr uint32_t kTermStride = (kTermBytes + kSlackBytes + 127) / 128 * 128;

template <int EPI>
constexpr int tile_threads() { return (3 + EPI) * 32; }
template <int EPI>
constexpr size_t tile_smem_bytes() {
    return 1024 + kPipeBytes + static_cast<size_t>(EPI) * 32 * kSlots * 8 + kTermBufs * kTermStride + 512;
}

__device__ __forceinline__ bool tile_extreme(float x2) { return (x2 > 0.0f && x2 < 0x1p-100f) || !(x2 < 0x1p100f); }

// Tiles are walked in groups of group_n base tiles, within which the query
// tile changes slowest: a base tile comes from HBM once and from L2 for every
// later query tile, and a query tile is loaded once per group. With `scout`
// there is one group, and each query tile meets its first `scout` base tiles
// twice, the first time with in_scout set. The walk is a counter per role
// (divisions only where it starts: finding every tile by division cost the
// epilogue as many instructions as reading the tile).
struct TileWalk {
    int mt, nt, left;   // left: base tiles of this query tile still to come, this one included
    int base, gsize;    // the group
    bool in_scout;
    __device__ __forceinline__ TileWalk(int t, const TileArgs& a) {
        if (a.scout) {
            mt = t / (a.ntiles + a.scout);
            const int rem = t - mt * (a.ntiles + a.scout);
            base = 0;
            gsize = a.ntiles;
            in_scout = rem < a.scout;
            nt = in_scout ? rem : rem - a.scout;
        } else {
            const int group = t / (a.mtiles * a.group_n);
            const int rem = t - group * a.mtiles * a.group_n;
            base = group * a.group_n;
            gsize = min(a.group_n, a.ntiles - base);
            mt = rem / gsize;
            nt = base + (rem - mt * gsize);
            in_scout = false;
        }
        left = in_scout ? a.scout - nt : base + gsize - nt;
    }
    __device__ __forceinline__ void next(const TileArgs& a) {
        ++nt;
        if (--left > 0) return;
        if (in_scout) {   // the same query tile again, in earnest
            in_scout = false;
            nt = base;
            left = gsize;
            return;
        }
        if (++mt == a.mtiles) {
            mt = 0;
            base += gsize;
            gsize = min(a.group_n, a.ntiles - base);
        }
        nt = base;
        in_scout = a.scout > 0;
        left = in_scout ? a.scout : gsize;
    }
};

__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// (bits, row) into the slot at shared address sp, which then moves on by
// `step`, when the float of `bits` is at most thr: predicated, no branch.
__device__ __forceinline__ void keep_below(uint32_t bits, uint32_t row, float thr, uint32_t& sp, uint32_t step) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.le.f32 p, %4, %3;\n\t"
        "@p st.shared.v2.b32 [%0], {%1, %2};\n\t"
        "@p add.u32 %0, %0, %5;\n\t}"
        : "+r"(sp)
        : "r"(bits), "r"(row), "f"(thr), "f"(__uint_as_float(bits)), "r"(step)
        : "memory");
}

// Warp 0 loads by TMA, warps 1 and 2 issue the MMAs of one query half each,
// the other EPI warps read the accumulators. 256 x 128 tiles: a base row that
// comes from L2 serves 256 queries (32 KB a tile of 128 dims; a 128 x 256
// tile needs 64 KB), and four halves fill TMEM, so that the epilogue of one
// tile runs under the MMAs of the next. Bound by the epilogue: 131,072 queries
// against 4,096 / 16,384 rows of 128 dims in 220 / 605 us (624 / 909 TFLOP/s
// counted once, the scout tiles on top), 156 / 507 us if no row passed and 117
// / 378 us with an epilogue that reads nothing; 768 dims 786 us (1,050
// TFLOP/s), there bound by L2, as both operands are streamed.
template <int EPI, int MODE>
__global__ void __launch_bounds__(tile_threads<EPI>(), 1)
    k_tile(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TileArgs a) {
    static_assert(EPI == 8 || EPI == 16, "8 or 16 epilogue warps");
    using namespace sm100;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const TilePipe pipe(a.kblocks, a.mtiles);
    const int S = pipe.stages;
    uint8_t* sA = base;                       // resident: two query tiles
    uint8_t* ring = base + pipe.ring_at;
    uint2* slots = reinterpret_cast<uint2*>(base + kPipeBytes);                        // [kSlots][EPI * 32]
    uint8_t* terms = reinterpret_cast<uint8_t*>(slots + static_cast<size_t>(EPI) * 32 * kSlots);   // [kTermBufs]
    uint64_t* bars = reinterpret_cast<uint64_t*>(terms + kTermBufs * kTermStride);
    uint64_t* full_r = bars;                  // [S] TMA -> MMA
    uint64_t* empty_r = bars + kMaxStages;    // [S] MMA -> TMA
    uint64_t* full_a = bars + 2 * kMaxStages;       // [2] TMA -> MMA
    uint64_t* empty_a = full_a + 2;                 // [2] MMA -> TMA
    uint64_t* tfull = full_a + 4;                   // [2 accumulators][2 halves] MMA -> epilogue
    uint64_t* tempty = full_a + 8;                  // [2][2] epilogue -> MMA
    uint64_t* mma_done = full_a + 12;               // [2] teardown
    uint64_t* full_x = full_a + 14;                 // [kTermBufs] TMA -> epilogue
    uint64_t* empty_x = full_x + kTermBufs;         // [kTermBufs] epilogue -> TMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty_x + kTermBufs);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (warp-uniform)
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full_r[s], 1);
            mbar_init(&empty_r[s], 2);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full_a[b], 1);
            mbar_init(&empty_a[b], 2);
            mbar_init(&mma_done[b], 1);
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], EPI / 2);
        }
        for (int b = 0; b < kTermBufs; ++b) {
            mbar_init(&full_x[b], 1);
            mbar_init(&empty_x[b], EPI);
        }
        *abort = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int total = a.mtiles * (a.ntiles + a.scout);
    const int per = (total + gridDim.x - 1) / gridDim.x;   // this CTA's tiles: [t_begin, t_end)
    const int t_begin = min(total, static_cast<int>(blockIdx.x) * per), t_end = min(total, t_begin + per);
    // What the loader and the MMA warps do between two barriers is not hidden by
    // the copies and MMAs they issue, so it is kept short: ring positions and
    // parities are carried (a division by the ring's length per K block held the
    // whole kernel to 1.1k cycles a block), the warps run converged and one elected
    // lane issues (addresses and descriptors stay in uniform registers: 179 ns a
    // K block of 4 MMAs against 310 ns from a branch on the lane index, of which
    // the MMAs are 136), and each half of the query tile has its own MMA warp.
    auto fail = [&] {
        *abort = 1;
        if (lane == 0) atomicExch(a.err, 2);
    };
    if (warp == 0) {
        int s = 0, cur_m = -1, ab = 1, xb = 0;
        uint32_t rpar = 1, apar = 0, xpar = 1;   // parities waited for: a fresh barrier passes the first wait for 1
        uint32_t loads = 0, aloads = 0, xloads = 0;
        bool ok = true;
        TileWalk w(t_begin, a);
        for (int t = t_begin; t < t_end && ok && !*abort; ++t, w.next(a)) {
            const int mt = w.mt, nt = w.nt;
            if (pipe.resident && mt != cur_m) {
                ab ^= 1;
                if (ab == 0) apar ^= 1;   // 1 for the first two loads
                if (!mbar_wait(&empty_a[ab], apar, abort)) {
                    fail();
                    break;
                }
                if (elect_one()) {
                    mbar_expect_tx(&full_a[ab], pipe.a_bytes);
                    for (int kb = 0; kb < a.kblocks; ++kb)
                        tma_load_2d(&tmA, sA + ab * pipe.a_bytes + kb * kABlock, &full_a[ab], kb * KA, mt * BM);
                }
                __syncwarp();
                ++aloads;
                cur_m = mt;
            }
            if (MODE != kStore) {   // the tile's row terms
                if (!mbar_wait(&empty_x[xb], xpar, abort)) {
                    fail();
                    break;
                }
                if (elect_one()) {
                    mbar_expect_tx(&full_x[xb], kTermBytes + (MODE == kNearest ? kSlackBytes : 0));
                    uint8_t* dst = terms + xb * kTermStride;
                    bulk_load(dst, a.xterm + a.n0 + static_cast<size_t>(nt) * BN, kTermBytes, &full_x[xb]);
                    if (MODE == kNearest)
                        bulk_load(dst + kTermBytes, a.run_slack + (a.n0 >> 5) + static_cast<size_t>(nt) * (BN / 32),
                                  kSlackBytes, &full_x[xb]);
                }
                __syncwarp();
                ++xloads;
                if (++xb == kTermBufs) {
                    xb = 0;
                    xpar ^= 1;
                }
            }
            for (int kb = 0; kb < a.kblocks; ++kb) {
                if (!mbar_wait(&empty_r[s], rpar, abort)) {
                    fail();
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    mbar_expect_tx(&full_r[s], pipe.stage_bytes);
                    uint8_t* dst = ring + s * pipe.stage_bytes;
                    tma_load_2d(&tmB, dst, &full_r[s], kb * KA, a.n0 + nt * BN);
                    if (!pipe.resident) tma_load_2d(&tmA, dst + kBBlock, &full_r[s], kb * KA, mt * BM);
                }
                __syncwarp();
                ++loads;
                if (++s == S) {
                    s = 0;
                    rpar ^= 1;
                }
            }
        }
        // no copy may land after the CTA is gone: wait for the last load of each buffer
        volatile int never = 0;
        for (int i = 0; i < S && static_cast<uint32_t>(i) < loads; ++i) {
            const uint32_t uses = (loads - i + S - 1) / S;   // of stage i
            mbar_wait(&full_r[i], (uses - 1) & 1, &never);
        }
        for (int b = 0; b < 2 && static_cast<uint32_t>(b) < aloads; ++b)
            mbar_wait(&full_a[b], ((aloads - b + 1) / 2 - 1) & 1, &never);
        for (int b = 0; b < kTermBufs && static_cast<uint32_t>(b) < xloads; ++b)
            mbar_wait(&full_x[b], ((xloads - b + kTermBufs - 1) / kTermBufs - 1) & 1, &never);
    } else if (warp <= 2) {
        const int h = warp - 1;
        const uint32_t idesc = idesc_f16_f32(128, BN);
        const uint64_t ring_d = sw128_desc(smem_u32(ring));
        const uint64_t a_d = sw128_desc(smem_u32(sA) + h * (kABlock / 2));
        const uint32_t stage_off = pipe.stage_bytes >> 4, abuf_off = pipe.a_bytes >> 4;   // (in descriptor units)
        int s = 0, cur_m = -1, ab = 1, acc = 0;
        uint32_t rpar = 0, apar = 1, tpar = 1;
        bool ok = true;
        TileWalk w(t_begin, a);
        for (int t = t_begin; t < t_end && ok && !*abort; ++t, w.next(a)) {
            const int mt = w.mt;
            if (pipe.resident && mt != cur_m) {
                if (cur_m >= 0 && elect_one()) mma_commit(&empty_a[ab]);   // free once its MMAs finish
                __syncwarp();
                ab ^= 1;
                if (ab == 0) apar ^= 1;   // 0 for the first two
                if (!mbar_wait(&full_a[ab], apar, abort)) {
                    fail();
                    break;
                }
                cur_m = mt;
            }
            if (!mbar_wait(&tempty[2 * acc + h], tpar, abort)) {
                fail();
                break;
            }
            const bool live = mt * BM + 128 * h < a.nq;   // (a half without queries is left out)
            const uint32_t td = tmem + acc * 256 + h * 128;
            for (int kb = 0; kb < a.kblocks; ++kb) {
                if (!mbar_wait(&full_r[s], rpar, abort)) {
                    fail();
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t bd = ring_d + s * stage_off;
                const uint64_t ad = pipe.resident ? a_d + ab * abuf_off + kb * (kABlock >> 4)
                                                  : bd + ((kBBlock + h * (kABlock / 2)) >> 4);
                const int ks1 = live ? min(4, a.ksteps - 4 * kb) : 0;
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)   // 32 bytes of K a step
                        if (ks < ks1) mma_f16(td, ad + 2 * ks, bd + 2 * ks, idesc, kb > 0 || ks > 0);
                    mma_commit(&empty_r[s]);
                    if (kb == a.kblocks - 1) mma_commit(&tfull[2 * acc + h]);
                }
                __syncwarp();
                if (++s == S) {
                    s = 0;
                    rpar ^= 1;
                }
            }
            if (!ok) break;
            acc ^= 1;
            if (acc == 0) tpar ^= 1;
        }
        // every MMA done before TMEM is freed
        volatile int never = 0;
        if (elect_one()) mma_commit(&mma_done[h]);
        __syncwarp();
        mbar_wait(&mma_done[h], 0, &never);
    } else {
        const int ew = warp - 3;      // 0..EPI-1
        const int quad = warp & 3;    // this warp's TMEM lanes: 32 * quad ..
        constexpr int kCols = BN / (EPI / 8);   // this warp's columns of its half
        constexpr int kRuns = kCols / 32;
        const int half = (ew >> 2) & 1, col0 = (ew >> 3) * kCols;
        uint2* slot = slots + ew * 32 + lane;   // entry i at slot[i * EPI * 32]
        uint32_t sp = smem_u32(slot);                                  // the next free place,
        const uint32_t room = sp + (kSlots - 3) * EPI * 32 * 8;        // the first with fewer than 4 after it
        int cur_m = -1, qi = 0;
        bool live = false;
        const float none = __int_as_float(0x7fffffff);   // (a lane without a query passes nothing)
        float qsl = 0.0f, thr = none;   // (lower bounds at or below thr pass)
        float2 mul2 = make_float2(0.0f, 0.0f);
        auto flush = [&] {
            const int cnt = static_cast<int>(sp - smem_u32(slot)) / (EPI * 32 * 8);
            const uint32_t pos = atomicAdd(&a.cand_count[qi], static_cast<uint32_t>(cnt));
            uint2* to = a.cand + static_cast<size_t>(qi) * a.cap + pos;
#pragma unroll 1
            for (int i = 0; i < cnt; ++i)
                if (pos + i < static_cast<uint32_t>(a.cap)) to[i] = slot[i * EPI * 32];
            sp = smem_u32(slot);
            // (no list holds more: the lane stops)
            if (MODE == kFilter && pos + cnt > static_cast<uint32_t>(kMaxCap)) thr = none;
        };
        auto leave = [&] {   // done with the query tile
            if (MODE == kStore) return;
            if (sp > smem_u32(slot)) flush();
            if (MODE == kNearest && live) atomicMin(&a.thr_key[qi], float_key(thr));
        };
        TileWalk w(t_begin, a);
        int acc = 0, xb = 0;
        uint32_t apar = 0, xpar = 0;
        for (int t = t_begin; t < t_end; ++t, w.next(a)) {
            const int mt = w.mt;
            if (mt != cur_m) {
                if (cur_m >= 0) leave();
                cur_m = mt;
                qi = mt * BM + half * 128 + quad * 32 + lane;
                live = qi < a.nq;
                const float mul = live && MODE != kStore ? -a.qmul[qi] : 0.0f;
                mul2 = make_float2(mul, mul);
                qsl = live && MODE == kNearest ? a.qslack[qi] : 0.0f;
                if (MODE != kStore) thr = live ? key_float(*reinterpret_cast<volatile uint32_t*>(a.thr_key + qi)) : none;
            }
            const float* sx = reinterpret_cast<const float*>(terms + xb * kTermStride) + col0;
            const float* sslack = reinterpret_cast<const float*>(terms + xb * kTermStride + kTermBytes) + col0 / 32;
            const bool ok = __all_sync(0xffffffffu, (MODE == kStore || mbar_wait(&full_x[xb], xpar, abort)) &&
                                                        mbar_wait(&tfull[2 * acc + half], apar, abort));
            if (!ok) {
                fail();
                break;
            }
            tc_fence_after();
            __syncwarp();   // (the TMEM loads below want a converged warp)
            // one run of 32 columns: its products in v. Lanes part ways in it (and where
            // one of them hands back): each call is followed by a __syncwarp
            auto run = [&](int r, uint32_t (&v)[32]) {
                if constexpr (MODE == kStore) {
                    const int c0 = w.nt * BN + col0 + 32 * r;
                    if (live) {
                        float* dst = a.store + static_cast<size_t>(qi) * a.ld + c0;
                        if (c0 + 32 <= a.ncols && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4)
                                *reinterpret_cast<float4*>(dst + j) =
                                    make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (c0 + j < a.ncols) dst[j] = __uint_as_float(v[j]);
                        }
                    }
                    return;
                }
                const float4* s4 = reinterpret_cast<const float4*>(sx + 32 * r);
                // the lower bounds (over the products), two a packed FMA, and
                // the smallest of every 4
                float gm[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const float4 x4 = s4[g];
                    const float2 l01 = __ffma2_rn(mul2, make_float2(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1])),
                                                  make_float2(x4.x, x4.y));
                    const float2 l23 = __ffma2_rn(mul2, make_float2(__uint_as_float(v[4 * g + 2]), __uint_as_float(v[4 * g + 3])),
                                                  make_float2(x4.z, x4.w));
                    gm[g] = fminf(min3(l01.x, l01.y, l23.x), l23.y);
                    v[4 * g] = __float_as_uint(l01.x);
                    v[4 * g + 1] = __float_as_uint(l01.y);
                    v[4 * g + 2] = __float_as_uint(l23.x);
                    v[4 * g + 3] = __float_as_uint(l23.y);
                }
                const float low = min3(min3(gm[0], gm[1], gm[2]), min3(gm[3], gm[4], gm[5]), fminf(gm[6], gm[7]));
                if (MODE == kNearest) {
                    thr = live ? fminf(thr, __fadd_ru(low, __fadd_ru(sslack[r], qsl))) : none;
                }
                if (w.in_scout || !__any_sync(0xffffffffu, low <= thr)) return;
                const uint32_t r0 = static_cast<uint32_t>(a.n0 + w.nt * BN + col0 + 32 * r);   // base row of v[0]
                // the groups in which some lane has one (one reduction: a vote and
                // a branch per group cost eight latencies)
                uint32_t groups = 0;
#pragma unroll
                for (int g = 0; g < 8; ++g) groups |= gm[g] <= thr ? 1u << g : 0u;
                groups = __reduce_or_sync(0xffffffffu, groups);
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    if (!((groups >> g) & 1u)) continue;
                    if (sp >= room) flush();
#pragma unroll
                    for (int j = 4 * g; j < 4 * g + 4; ++j) keep_below(v[j], r0 + j, thr, sp, EPI * 32 * 8);
                }
            };
            const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16) +
                                   static_cast<uint32_t>(acc * 256 + half * 128 + col0);
            auto hand_back = [&] {   // this warp's last read: the accumulator goes back before the work on it
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[2 * acc + half]);
            };
            if constexpr (EPI == 8) {
                // each run's load goes under the work on the run before it (64
                // registers, which 8 warps have and 16 do not)
                uint32_t va[32], vb[32];
                tmem_ld32_start(taddr, va);
#pragma unroll 1
                for (int r = 0; r < kRuns; r += 2) {
                    tmem_ld32_wait(va);
                    tmem_ld32_start(taddr + 32 * (r + 1), vb);
                    run(r, va);
                    __syncwarp();
                    tmem_ld32_wait(vb);
                    if (r + 2 < kRuns) tmem_ld32_start(taddr + 32 * (r + 2), va);
                    else hand_back();
                    run(r + 1, vb);
                    __syncwarp();
                }
            } else {
#pragma unroll 1
                for (int r = 0; r < kRuns; ++r) {
                    uint32_t v[32];
                    tmem_ld32(taddr + 32 * r, v);
                    if (r == kRuns - 1) hand_back();
                    run(r, v);
                    __syncwarp();
                }
            }
            acc ^= 1;
            if (acc == 0) apar ^= 1;
            if (MODE == kStore) continue;
            // (the warp's reads of the row terms are done)
            if (lane == 0) mbar_arrive(&empty_x[xb]);
            if (++xb == kTermBufs) {
                xb = 0;
                xpar ^= 1;
            }
        }
        if (cur_m >= 0) leave();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_free(tmem, kTmemCols);
    }
}

// ---- preparing rows ------------------------------------------------------------

// x 2^e rounded to f16 (one exact multiply when 2^e is a normal float)
__device__ __forceinline__ __half scaled_half(float x, int e) {
    const float y = (e >= -126 && e <= 127) ? __fmul_rn(x, __int_as_float((e + 127) << 23)) : ldexpf(x, e);
    return __float2half_rn(y);
}

// The exponent that puts the largest magnitude m into [2^13, 2^14).
__device__ __forceinline__ int lift_exp(float m) {
    int ex = 0;
    if (m > 0.0f) frexpf(m, &ex);
    return m > 0.0f ? 14 - ex : 0;
}

// The largest magnitude below 2^50 (rows holding a larger one are extreme) as
// its float bits, by one atomic per block.
__global__ void __launch_bounds__(256) k_tile_amax(const float* __restrict__ x, size_t n, uint32_t* __restrict__ amax) {
    float m = 0.0f;
    auto take = [&](float v) {
        const float b = fabsf(v);
        if (b < 0x1p50f) m = fmaxf(m, b);
    };
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t n4 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / 4 : 0;
    for (size_t i = t; i < n4; i += step) {
        const float4 v = reinterpret_cast<const float4*>(x)[i];
        take(v.x);
        take(v.y);
        take(v.z);
        take(v.w);
    }
    for (size_t i = 4 * n4 + t; i < n; i += step) take(x[i]);
    __shared__ float wm[8];
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = fmaxf(m, wm[w]);
        if (m > 0.0f) atomicMax(amax, __float_as_uint(m));   // (non-negative floats order as their bits)
    }
}

// Base rows to f16 with the shared exponent, and their squared norms. One warp
// per row, twice over a row that the first read leaves in L1.
__global__ void __launch_bounds__(256) k_tile_base(const float* __restrict__ x, size_t n, int d, int dpad,
                                                   const uint32_t* __restrict__ amax, __half* __restrict__ xh,
                                                   float* __restrict__ x2) {
    const size_t r = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const int e = lift_exp(__uint_as_float(*amax));
    const float* row = x + r * d;
    float s = 0.0f;
    for (int j = lane; j < d; j += 32) s = __fmaf_rn(row[j], row[j], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const bool zero = tile_extreme(s);
    for (int j = lane; j < dpad; j += 32)
        xh[r * dpad + j] = j < d && !zero ? scaled_half(row[j], e) : __float2half_rn(0.0f);
    if (lane == 0) x2[r] = s;
}

// Query rows to f16, each with its own exponent, and their squared norms.
__global__ void __launch_bounds__(256) k_tile_queries(const float* __restrict__ x, size_t n, int d, int dpad,
                                                      __half* __restrict__ xh, float* __restrict__ x2,
                                                      int* __restrict__ xe) {
    const size_t r = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const float* row = x + r * d;
    float s = 0.0f, mx = 0.0f;
    for (int j = lane; j < d; j += 32) {
        const float v = row[j];
        s = __fmaf_rn(v, v, s);
        mx = fmaxf(mx, fabsf(v));
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const bool zero = tile_extreme(s);
    const int e = zero ? 0 : lift_exp(mx);
    for (int j = lane; j < dpad; j += 32)
        xh[r * dpad + j] = j < d && !zero ? scaled_half(row[j], e) : __float2half_rn(0.0f);
    if (lane == 0) {
        x2[r] = s;
        xe[r] = e;
    }
}

// The bound's factors (top of the file).
struct TileBound {
    float mult;   // of acc
    float xc;     // xterm = xc |x|^2
    float c2;     // 2 c
    float g2;     // 2 g = g2 |q| M
    TileBound(int d, bool ip) {
        const double C = tile_error_factor(d);
        mult = ip ? 1.0f : 2.0f;
        xc = static_cast<float>(ip ? -0.5 * C : 1.0 - C);
        c2 = static_cast<float>(ip ? C : 2.0 * C);
        g2 = static_cast<float>((ip ? 2.0 : 4.0) * std::sqrt(double(d)) * std::ldexp(1.0, -37));
    }
};

// Each base row's part of the lower bound (+inf for rows that are refused,
// -inf for extreme ones, which always pass), and per 32 rows the slack that
// takes the smallest lower bound among them to an upper bound. The terms and norms of
// the sample (rows step apart) once more, side by side: read in place by every query's
// block they cost 10,000 queries 250 us. With `apart` the sample's rows are not to be
// returned again.
__global__ void __launch_bounds__(256) k_tile_terms(const float* __restrict__ sq, size_t n, size_t npad, TileBound b,
                                                    const uint64_t* __restrict__ allow,
                                                    const uint64_t* __restrict__ deny, float* __restrict__ xterm,
                                                    float* __restrict__ run_slack, uint32_t step, uint32_t sampled, bool apart,
                                                    float* __restrict__ sample_term, float* __restrict__ sample_sq) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    constexpr float kInf = __builtin_huge_valf();
    float s = 0.0f;
    if (i < n) {
        const float x2 = sq[i];
        const bool ex = tile_extreme(x2);
        const bool refused = (allow && !((allow[i >> 6] >> (i & 63)) & 1ull)) ||
                             (deny && ((deny[i >> 6] >> (i & 63)) & 1ull));
        const float term = refused ? kInf : ex ? -kInf : __fmul_rn(b.xc, x2);
        const uint32_t j = static_cast<uint32_t>(i) / step;
        const bool in = j < sampled && j * step == i;
        xterm[i] = in && apart ? kInf : term;
        if (in) {
            sample_term[j] = term;
            sample_sq[j] = x2;
        }
        s = ex ? kInf : __fmul_ru(b.c2, x2);
    } else if (i < npad) {
        xterm[i] = kInf;
    }
    s = warp_max(s);
    if ((threadIdx.x & 31) == 0 && i < npad) run_slack[i >> 5] = s;
}

// Per query: the factor that takes acc to the row's scale, the slack, an open
// threshold and an empty candidate list. An extreme query's list counts as
// overflowed from the start.
__global__ void k_tile_open(const float* __restrict__ q2, const int* __restrict__ qexp, int nq, TileBound b,
                            const uint32_t* __restrict__ amax, int cap, float* __restrict__ qmul,
                            float* __restrict__ qslack, uint32_t* __restrict__ thr_key, uint32_t* __restrict__ count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    const float s = q2[i], M = __uint_as_float(*amax);
    const bool ex = tile_extreme(s);
    qmul[i] = ldexpf(b.mult, -(qexp[i] + lift_exp(M)));
    qslack[i] = ex ? 0.0f : __fadd_ru(__fmul_ru(b.c2, s), __fmul_ru(b.g2, __fmul_ru(__fsqrt_ru(s), M)));
    thr_key[i] = float_key(ex ? -kOpen : kOpen);
    count[i] = ex ? static_cast<uint32_t>(cap) + 1 : 0u;
}

// One warp per query: of its candidates, those whose lower bound is at most
// the smallest upper bound. A single one is the nearest row; several are
// scored exactly, 8 at a time by 4-lane groups (even dim at 8-byte alignment,
// kG = 4) or 4 at a time by 8-lane groups, and the smallest (score, row) wins.
// An overflowed list goes to redo.
template <int kG>
__global__ void __launch_bounds__(256) k_tile_pick(const float* __restrict__ q, int d, const float* __restrict__ rows,
                                                   int nq, const uint32_t* __restrict__ count,
                                                   const uint2* __restrict__ cand, int cap,
                                                   const uint32_t* __restrict__ thr_key, uint32_t first,
                                                   uint32_t* __restrict__ label, uint32_t* __restrict__ redo,
                                                   uint32_t* __restrict__ nredo) {
    const int qi = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (qi >= nq) return;
    const uint32_t cnt = count[qi];
    const float T = key_float(thr_key[qi]);
    const uint2* c = cand + static_cast<size_t>(qi) * cap;
    const float* qv = q + static_cast<size_t>(qi) * d;
    constexpr int kPer = 32 / kG;   // candidates scored together
    uint64_t best = ~0ull;
    uint32_t one = 0, passed = 0;
    if (cnt <= static_cast<uint32_t>(cap)) {
        for (uint32_t b = 0; b < cnt; b += 32) {
            const uint2 e = b + lane < cnt ? c[b + lane] : make_uint2(0x7f800000u, 0u);
            const unsigned in = __ballot_sync(0xffffffffu, b + lane < cnt && __uint_as_float(e.x) <= T);
            passed += __popc(in);
            if (in) one = __shfl_sync(0xffffffffu, e.y, __ffs(in) - 1);
        }
        for (uint32_t b = 0; passed > 1 && b < cnt; b += 32) {
            const uint2 e = b + lane < cnt ? c[b + lane] : make_uint2(0x7f800000u, 0u);
            unsigned in = __ballot_sync(0xffffffffu, b + lane < cnt && __uint_as_float(e.x) <= T);
            while (in) {
                // this lane group's candidate: the set bit of its rank
                unsigned m = in;
                for (int g = 0; g < lane / kG && m; ++g) m &= m - 1;
                const bool act = m != 0;
                const uint32_t row = __shfl_sync(0xffffffffu, e.y, act ? __ffs(m) - 1 : 0);
                const float* rp = rows + static_cast<size_t>(row) * d;
                const float s = kG == 4 ? exact_avx2_group4<true>(qv, rp, d) : exact_avx2_group8<true, true>(qv, rp, d);
                const uint64_t key = act ? (static_cast<uint64_t>(float_key_eq0(s)) << 32) | row : ~0ull;
                best = key < best ? key : best;
                for (int g = 0; g < kPer && in; ++g) in &= in - 1;
            }
        }
    }
    if (passed > 1) {
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other < best ? other : best;
        }
        one = static_cast<uint32_t>(best);
    }
    if (lane == 0) {
        if (passed > 0) label[qi] = one;
        else redo[atomicAdd(nredo, 1u)] = first + qi;
    }
}

// ---- the k nearest ----------------------------------------------------------------
//
// The products of a sample of the rows, at equal steps, are stored, and each
// query's threshold is the k-th smallest upper bound among them. (The first rows
// would do as well where rows are stored in random order. Where they are not, by
// cluster or by time, what is near would meet a threshold from rows that are far.)
// The sample's rows below it open the query's candidate list; the other
// rows are taken in chunks of growing size: the engine appends
// the rows whose lower bound is below the threshold, and a cut per query takes
// the threshold to the k-th smallest upper bound of all its candidates and
// drops those above. Only what is left at the end is scored exactly.

// A threshold at or just above the k-th smallest of n upper bounds (kOpen when
// fewer than k are finite), by one block; ub: the bounds in shared memory. They
// are counted into 1,024 equal intervals of their range, and the interval that
// holds the k-th is cut again while it holds many more than are wanted; the
// threshold is the largest bound in the last one. (Intervals of the bounds'
// ordered bits took in 6 times too many when the range crosses zero.)
struct CutScratch {
    int hist[kKeyHist];
    float lo[8], hi[8];
    int fin[8], pick[3], count;
};
__device__ __forceinline__ float cut_threshold(const float* ub, int n, int k, CutScratch& s) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    constexpr float kInf = __builtin_huge_valf();
    if (threadIdx.x == 0) s.count = 0;
    // the range and number of the bounds that in() admits
    auto range = [&](auto in, float& lo, float& hi, int& fin) {
        lo = kInf;
        hi = -kInf;
        fin = 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float u = ub[i];
            if (in(u)) {
                lo = fminf(lo, u);
                hi = fmaxf(hi, u);
                ++fin;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        fin = __reduce_add_sync(0xffffffffu, fin);
        __syncthreads();   // (the scratch of an earlier call is read)
        if (lane == 0) {
            s.lo[warp] = lo;
            s.hi[warp] = hi;
            s.fin[warp] = fin;
        }
        for (int t = threadIdx.x; t < kKeyHist; t += blockDim.x) s.hist[t] = 0;
        __syncthreads();
        fin = 0;
        for (int w = 0; w < nw; ++w) {
            lo = fminf(lo, s.lo[w]);
            hi = fmaxf(hi, s.hi[w]);
            fin += s.fin[w];
        }
    };
    float lo, hi;
    int fin, need = k;
    range([](float u) { return u <= kOpen; }, lo, hi, fin);
    if (fin < k) return kOpen;   // (block-uniform, as everything below)
    for (int level = 0; level < 3; ++level) {
        const float scale = __fdiv_rn(static_cast<float>(kKeyBins), __fsub_rn(hi, lo));
        if (fin - need <= k / 8 || !(scale > 0.0f && scale <= kOpen)) break;
        const float from = lo, to = hi;
        // (monotone in u: the subtraction, the product and the conversion are)
        auto bin = [&](float u) { return min(kKeyBins - 1, __float2int_rd(__fmul_rn(__fsub_rn(u, from), scale))); };
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float u = ub[i];
            if (u >= from && u <= to) {
                const int b = bin(u);
                atomicAdd(&s.hist[b + (b >> 5)], 1);
            }
        }
        __syncthreads();
        if (warp == 0) {   // lane l owns bins 32 l .. 32 l + 31
            int own = 0;
#pragma unroll 8
            for (int b = 0; b < 32; ++b) own += s.hist[33 * lane + b];
            int incl = own;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int excl = incl - own;
            if (excl < need && need <= incl) {
                int acc = excl;
                for (int b = 0; b < 32; ++b) {
                    const int c = s.hist[33 * lane + b];
                    if (acc + c >= need) {
                        s.pick[0] = 32 * lane + b;
                        s.pick[1] = acc;
                        break;
                    }
                    acc += c;
                }
            }
        }
        __syncthreads();
        const int pick = s.pick[0];
        need -= s.pick[1];
        range([&](float u) { return u >= from && u <= to && bin(u) == pick; }, lo, hi, fin);
    }
    return hi;   // need of the bounds in [lo, hi] and k of all are at or below it
}

__device__ __forceinline__ float upper_bound(float lb, float x2, float c2, float qslack) {
    // (an extreme row's lower bound says nothing about where it is)
    return tile_extreme(x2) ? __builtin_huge_valf() : __fadd_ru(lb, __fadd_ru(__fmul_ru(c2, x2), qslack));
}

// The key of a threshold that no row passes, extreme ones included.
constexpr uint32_t kClosedKey = 0xFFFFFFFFu;   // (a NaN)

// One block per query over the stored products of a sample of ncols rows: its
// threshold, and with `step` (0: the threshold alone) the rows at or below it, which
// are `step` apart. lbs, ub: ncols floats of shared memory each.
__global__ void __launch_bounds__(256) k_tile_seed(const float* __restrict__ acc, size_t ld, int ncols,
                                                   const float* __restrict__ xterm, const float* __restrict__ sq,
                                                   float c2, const float* __restrict__ qmul,
                                                   const float* __restrict__ qslack, int k, int cap, uint32_t step,
                                                   uint32_t* __restrict__ thr_key, uint32_t* __restrict__ count,
                                                   uint2* __restrict__ cand) {
    extern __shared__ __align__(16) uint8_t sm_raw[];
    __shared__ CutScratch s;
    const int qi = blockIdx.x;
    if (count[qi] > static_cast<uint32_t>(cap)) {   // an extreme query
        __syncthreads();
        if (threadIdx.x == 0) {
            count[qi] = kGivenUp;
            thr_key[qi] = kClosedKey;
        }
        return;
    }
    float* lbs = reinterpret_cast<float*>(sm_raw);
    float* ub = lbs + ncols;
    const float* row = acc + static_cast<size_t>(qi) * ld;
    const float mul = -qmul[qi], qs = qslack[qi];
    for (int j = threadIdx.x; j < ncols; j += blockDim.x) {
        const float lb = __fmaf_rn(mul, row[j], xterm[j]);
        lbs[j] = lb;
        // (refused rows: +inf)
        ub[j] = lb <= kOpen ? upper_bound(lb, sq[j], c2, qs) : __builtin_huge_valf();
    }
    __syncthreads();
    const float T = cut_threshold(ub, ncols, k, s);
    if (step == 0) {
        if (threadIdx.x == 0) thr_key[qi] = float_key(T);
        return;
    }
    const int lane = threadIdx.x & 31;
    for (int j0 = 0; j0 < ncols; j0 += blockDim.x) {   // (trip count block-uniform)
        const int j = j0 + threadIdx.x;
        const float lb = j < ncols ? lbs[j] : __builtin_huge_valf();
        const unsigned in = __ballot_sync(0xffffffffu, lb <= T);
        if (in == 0) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s.count, __popc(in));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(in & ((1u << lane) - 1));
        if (lb <= T && at < cap)
            cand[static_cast<size_t>(qi) * cap + at] = make_uint2(__float_as_uint(lb), static_cast<uint32_t>(j) * step);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        count[qi] = static_cast<uint32_t>(s.count);
        thr_key[qi] = float_key(T);
    }
}

// The candidates of one query at or below their k-th smallest upper bound,
// compacted to the front of list[] in shared memory (by one block; n of them
// on entry); returns how many, and the threshold in T. ub: n floats of scratch.
__device__ __forceinline__ int cut_list(uint2* list, float* ub, int n, int k, const float* __restrict__ sq, float c2,
                                        float qs, CutScratch& s, float& T) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        ub[i] = upper_bound(__uint_as_float(list[i].x), sq[list[i].y], c2, qs);
    __syncthreads();
    T = cut_threshold(ub, n, k, s);
    const int lane = threadIdx.x & 31;
    int kept = 0;
    for (int i0 = 0; i0 < n; i0 += blockDim.x) {   // (trip count block-uniform)
        const int i = i0 + threadIdx.x;
        const uint2 e = i < n ? list[i] : make_uint2(0x7f800000u, 0u);
        const bool in = i < n && __uint_as_float(e.x) <= T;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        __syncthreads();   // this round's entries are read before any is overwritten
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&s.count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1));
        if (in) list[at] = e;   // (at < i0 + blockDim.x: only read entries)
    }
    __syncthreads();
    kept = s.count;
    return kept;
}

// The stored products of the sample, and what bounds take from its rows.
struct Sample {
    const float* acc;   // per query, ld apart
    size_t ld;
    int ncols;
    const float *xterm, *sq;
};

// Whether a sweep would settle a list that overflowed under the threshold of key
// `was`, with cnt rows counted: its list holds them all, or a lower threshold is to be
// had, from the entries the list did take or from the nearest row of the sample (not
// so where more rows tie than any list holds). By one block; list, ub: cap entries of
// shared memory each. (Not inlined: it is rare, and its registers cost the kernels
// around it 3 to 8 % of the search.)
__device__ __noinline__ bool worth_a_sweep(const uint2* mine, uint32_t cnt, uint32_t was, const float* acc, Sample sm,
                                           float qmul, float qs, uint2* list, float* ub, int cap, int k,
                                           const float* __restrict__ sq, float c2, CutScratch& s) {
    if (cnt <= static_cast<uint32_t>(kMaxCap)) return true;   // (block-uniform)
    const float T = key_float(was);
    bool lower = false;
    for (int j = threadIdx.x; j < sm.ncols; j += blockDim.x) {
        const float lb = __fmaf_rn(-qmul, acc[j], sm.xterm[j]);
        lower |= lb <= kOpen && upper_bound(lb, sm.sq[j], c2, qs) < T;
    }
    if (__syncthreads_or(lower)) return true;
    for (int i = threadIdx.x; i < cap; i += blockDim.x) list[i] = mine[i];
    __syncthreads();
    float best;
    cut_list(list, ub, cap, k, sq, c2, qs, s, best);
    return best < T;
}

// After a chunk, one block per query: the list cut, its threshold lowered (not while the
// list holds fewer than k rows).
__global__ void __launch_bounds__(128) k_tile_cut(const float* __restrict__ sq, float c2,
                                                  const float* __restrict__ qslack, int k, int cap,
                                                  uint32_t* __restrict__ thr_key, uint32_t* __restrict__ count,
                                                  uint2* __restrict__ cand) {
    extern __shared__ __align__(16) uint8_t sm_raw[];
    __shared__ CutScratch s;
    const int qi = blockIdx.x;
    const uint32_t cnt = count[qi], was = thr_key[qi];
    if (cnt > static_cast<uint32_t>(cap)) return;   // overflowed: only counted on
    const int n = static_cast<int>(cnt);
    uint2* list = reinterpret_cast<uint2*>(sm_raw);
    float* ub = reinterpret_cast<float*>(list + cap);
    uint2* mine = cand + static_cast<size_t>(qi) * cap;
    for (int i = threadIdx.x; i < n; i += blockDim.x) list[i] = mine[i];
    __syncthreads();
    float T;
    const int kept = cut_list(list, ub, n, k, sq, c2, qslack[qi], s, T);
    for (int i = threadIdx.x; i < kept; i += blockDim.x) mine[i] = list[i];
    if (threadIdx.x == 0) {
        count[qi] = static_cast<uint32_t>(kept);
        thr_key[qi] = min(was, float_key(T));
    }
}

// After a sweep over every row, one block per query. A list that held what
// passed is cut and closed. In one that overflowed, the entries it did take are
// rows like any others, so the k-th smallest of their upper bounds is a threshold: with
// that one, where it is lower, the list is opened again (*open counts those);
// otherwise, or after the last sweep, it is given up.
__global__ void __launch_bounds__(128) k_tile_sweep_cut(const float* __restrict__ sq, float c2,
                                                        const float* __restrict__ qslack, int k, int cap, bool last,
                                                        uint32_t* __restrict__ thr_key, uint32_t* __restrict__ count,
                                                        uint2* __restrict__ cand, uint32_t* __restrict__ open) {
    extern __shared__ __align__(16) uint8_t sm_raw[];
    __shared__ CutScratch s;
    const int qi = blockIdx.x;
    const uint32_t was = thr_key[qi], cnt = count[qi];
    if (was == kClosedKey) return;
    const bool held = cnt <= static_cast<uint32_t>(cap);
    const int n = held ? static_cast<int>(cnt) : cap;
    uint2* list = reinterpret_cast<uint2*>(sm_raw);
    float* ub = reinterpret_cast<float*>(list + cap);
    uint2* mine = cand + static_cast<size_t>(qi) * cap;
    for (int i = threadIdx.x; i < n; i += blockDim.x) list[i] = mine[i];
    __syncthreads();
    float T;
    const int kept = cut_list(list, ub, n, k, sq, c2, qslack[qi], s, T);
    const bool again = !held && !last && float_key(T) < was;
    if (held)
        for (int i = threadIdx.x; i < kept; i += blockDim.x) mine[i] = list[i];
    if (threadIdx.x == 0) {
        thr_key[qi] = again ? float_key(T) : kClosedKey;
        count[qi] = held ? static_cast<uint32_t>(kept) : again ? 0u : kGivenUp;
        if (again) atomicAdd(open, 1u);
    }
}

// At the end, one block per query: the list cut, the rows left scored exactly
// (a lane group of kG per row: 4 for an even dim at 8-byte alignment, else 8), and
// the k smallest by (score, row) written in order. Up to 512 keys are ranked
// over per-warp register-sorted runs (one barrier), more sorted by the block.
template <int kG>
__global__ void __launch_bounds__(256, 6) k_tile_finish(const float* __restrict__ q, int d, const float* __restrict__ rows,
                                                     bool ip, const float* __restrict__ sq, float c2,
                                                     const float* __restrict__ qslack, int k, int cap,
                                                     const uint32_t* __restrict__ count,
                                                     const uint32_t* __restrict__ thr_key,
                                                     const uint2* __restrict__ cand, Sample sample,
                                                     const float* __restrict__ qmul, uint32_t first,
                                                     uint64_t* __restrict__ out_key, uint32_t* __restrict__ out_slot,
                                                     uint32_t* __restrict__ redo, uint32_t redo_end,
                                                     uint32_t* __restrict__ nredo) {
    extern __shared__ __align__(16) uint8_t sm_raw[];
    __shared__ CutScratch s;
    const int qi = blockIdx.x;
    const uint32_t cnt = count[qi];
    const int n = static_cast<int>(cnt);
    uint2* list = reinterpret_cast<uint2*>(sm_raw);
    float* ub = reinterpret_cast<float*>(list + cap);
    const uint2* mine = cand + static_cast<size_t>(qi) * cap;
    if (cnt > static_cast<uint32_t>(cap)) {   // to the front of redo[] to be swept, to its end where that would not help
        const bool sweep =
            cnt != kGivenUp && worth_a_sweep(mine, cnt, thr_key[qi], sample.acc + static_cast<size_t>(qi) * sample.ld,
                                             sample, qmul[qi], qslack[qi], list, ub, cap, k, sq, c2, s);
        if (threadIdx.x == 0) {
            if (sweep) redo[atomicAdd(nredo, 1u)] = first + qi;
            else redo[redo_end - 1 - atomicAdd(nredo + 1, 1u)] = first + qi;
        }
        return;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) list[i] = mine[i];
    __syncthreads();
    float T;
    const int m = cut_list(list, ub, n, k, sq, c2, qslack[qi], s, T);
    // exact keys over the list, entry by entry (a group reads its row first)
    uint64_t* ekey = reinterpret_cast<uint64_t*>(list);
    const float* qv = q + static_cast<size_t>(qi) * d;
    const int ngrp = blockDim.x / kG, grp = threadIdx.x / kG;
    for (int i0 = 0; i0 < m; i0 += ngrp) {   // (block-uniform)
        const int i = i0 + grp;
        const bool act = i < m;
        const uint32_t row = act ? list[i].y : 0u;   // idle groups score row 0 unused
        const float* rp = rows + static_cast<size_t>(row) * d;
        float sc;
        if constexpr (kG == 4) sc = ip ? -exact_avx2_group4<false>(qv, rp, d) : exact_avx2_group4<true>(qv, rp, d);
        else sc = ip ? -exact_avx2_group8<false, true>(qv, rp, d) : exact_avx2_group8<true, true>(qv, rp, d);
        __syncwarp();
        if (act && threadIdx.x % kG == 0) ekey[i] = (static_cast<uint64_t>(float_key_eq0(sc)) << 32) | row;
    }
    uint64_t* ok = out_key + static_cast<size_t>(qi) * k;
    uint32_t* os = out_slot + static_cast<size_t>(qi) * k;
    const int got = min(m, k);
    for (int i = got + threadIdx.x; i < k; i += blockDim.x) {
        ok[i] = ~0ull;
        os[i] = 0xFFFFFFFFu;
    }
    __syncthreads();
    if (m <= 512) {   // (block-uniform)
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int n_w = max(0, min(64, m - 64 * warp));
        if (n_w > 0) warp_sort_keys_reg<2>(ekey + 64 * warp, n_w);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = 32 * i + lane;
            if (e >= n_w) continue;
            const uint64_t kk = ekey[64 * warp + e];
            int rank = 0;
            for (int w = 0; 64 * w < m; ++w) {
                const int len = min(64, m - 64 * w);
                const uint64_t* rw = ekey + 64 * w;
                int pos = 0;
#pragma unroll
                for (int step = 64; step > 0; step >>= 1)
                    if (pos + step <= len && rw[pos + step - 1] < kk) pos += step;
                rank += pos;
            }
            if (rank < k) {
                ok[rank] = kk;
                os[rank] = static_cast<uint32_t>(kk);
            }
        }
        return;
    }
    const int np = next_pow2(m);   // (at most the list's power-of-two cap)
    for (int i = m + threadIdx.x; i < np; i += blockDim.x) ekey[i] = ~0ull;
    bitonic_sort_keys(ekey, np);
    for (int i = threadIdx.x; i < got; i += blockDim.x) {
        ok[i] = ekey[i];
        os[i] = static_cast<uint32_t>(ekey[i]);
    }
}

// ---- launching ------------------------------------------------------------------

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    });
    require(fn != nullptr, "cuTensorMapEncodeTiled is not available", kCudaError);
    return fn;
}

// f16 rows (dpad elements, row stride dpad * 2 bytes, or `step` such rows) read as boxes of 64 x box_rows,
// 128-byte swizzle.
CUtensorMap make_map(const void* ptr, size_t rows, int dpad, int box_rows, size_t step = 1) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(dpad), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(dpad) * 2 * step};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(KA), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
                                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    require(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed", kCudaError);
    return m;
}

// The epilogue's warp count is the schedule choice: 8 (each warp 128 columns
// of its 32 queries) or 16 (64 columns each). On the first launch of a problem
// (mode, K blocks, query and base tiles by their power of two) with at least 8
// tiles per SM, both are timed twice on the launch's own inputs and the faster
// kept for the rest of the process; save() keeps what the launch changes,
// reset() puts it back before each further run, and the last run's is the
// launch's result. Both give the same results. Launches that must not wait on
// the host use the problem's pick if there is one, else 16.
std::mutex g_tune_mu;
std::map<uint64_t, int> g_tuned;   // problem key -> epilogue warps
std::atomic<int> g_tune_on{1}, g_tune_last{8}, g_tune_force{0};

template <int EPI, int MODE>
void launch_epi(const CUtensorMap& tmA, const CUtensorMap& tmB, const TileArgs& a, cudaStream_t st) {
    allow_large_smem<k_tile<EPI, MODE>>();
    const int tiles = a.mtiles * (a.ntiles + a.scout);
    const int ctas = std::min(tiles, a.ctas > 0 ? std::min(a.ctas, sm_count()) : sm_count());
    k_tile<EPI, MODE><<<static_cast<unsigned>(ctas), tile_threads<EPI>(), tile_smem_bytes<EPI>(), st>>>(tmA, tmB, a);
    QG_LAUNCH_CHECK();
}

template <int MODE>
void launch_as(int epi, const CUtensorMap& tmA, const CUtensorMap& tmB, const TileArgs& a, cudaStream_t st) {
    if (epi == 16) launch_epi<16, MODE>(tmA, tmB, a, st);
    else launch_epi<8, MODE>(tmA, tmB, a, st);
    g_tune_last.store(epi);
}

template <int MODE, class Save, class Reset>
void launch_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, const TileArgs& a, cudaStream_t st, bool may_tune,
                 Save save, Reset reset) {
    if (const int f = g_tune_force.load()) {
        launch_as<MODE>(f, tmA, tmB, a, st);
        return;
    }
    const uint64_t key = (static_cast<uint64_t>(MODE) << 48) | (static_cast<uint64_t>(a.kblocks) << 40) |
                         (static_cast<uint64_t>(next_pow2(a.mtiles)) << 20) | static_cast<uint64_t>(next_pow2(a.ntiles));
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        const auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            launch_as<MODE>(it->second, tmA, tmB, a, st);
            return;
        }
    }
    if (!may_tune || !g_tune_on.load() || static_cast<long long>(a.mtiles) * a.ntiles < 8ll * sm_count()) {
        launch_as<MODE>(16, tmA, tmB, a, st);
        return;
    }
    save();
    cudaEvent_t e0, e1;
    QG_CUDA(cudaEventCreate(&e0));
    QG_CUDA(cudaEventCreate(&e1));
    constexpr int kCand[2] = {8, 16};
    float fastest[2] = {0.0f, 0.0f};
    for (int round = 0; round < 2; ++round)
        for (int c = 0; c < 2; ++c) {
            if (round + c > 0) reset();
            QG_CUDA(cudaEventRecord(e0, st));
            launch_as<MODE>(kCand[c], tmA, tmB, a, st);
            QG_CUDA(cudaEventRecord(e1, st));
            QG_CUDA(cudaEventSynchronize(e1));
            float ms = 0.0f;
            QG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            if (round == 0 || ms < fastest[c]) fastest[c] = ms;
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    std::lock_guard<std::mutex> g(g_tune_mu);
    g_tuned[key] = fastest[1] < fastest[0] ? 16 : 8;
}

unsigned blocks_of(size_t n, size_t per = 256) { return static_cast<unsigned>(ceil_div(std::max<size_t>(1, n), per)); }

} // namespace

void set_tile_autotune(int on) { g_tune_on.store(on); }
int tile_autotune() { return g_tune_on.load(); }
int64_t tile_tuned_problems() {
    std::lock_guard<std::mutex> g(g_tune_mu);
    return static_cast<int64_t>(g_tuned.size());
}
int tile_last_epilogue_warps() { return g_tune_last.load(); }
void set_tile_epilogue_warps(int warps) { g_tune_force.store(warps); }
int tile_epilogue_warps() { return g_tune_force.load(); }

double tile_error_factor(int dim) { return std::ldexp(1.0, -10) + std::ldexp(1.0, -13) + dim * std::ldexp(1.0, -21); }

bool tile_supported(int dim) { return dim >= 1 && dim <= kMaxDim; }

void tile_prepare_queries(const float* rows, size_t n, int dim, TileQueries& out, cudaStream_t st) {
    require(tile_supported(dim), "the tensor-core path does not support this dimension", kUnsupported);
    out.n = n;
    out.dim = dim;
    out.dpad = (dim + 7) & ~7;
    out.f16.alloc(std::max<size_t>(1, n * out.dpad), st);
    out.sq.alloc(std::max<size_t>(1, n), st);
    out.exps.alloc(std::max<size_t>(1, n), st);
    if (n == 0) return;
    k_tile_queries<<<blocks_of(n * 32), 256, 0, st>>>(rows, n, dim, out.dpad, reinterpret_cast<__half*>(out.f16.get()),
                                                      out.sq.get(), out.exps.get());
    QG_LAUNCH_CHECK();
}

void tile_prepare_base(const float* rows, size_t n, int dim, TileBase& out, cudaStream_t st) {
    require(tile_supported(dim), "the tensor-core path does not support this dimension", kUnsupported);
    out.n = n;
    out.dim = dim;
    out.dpad = (dim + 7) & ~7;
    out.f16.alloc(std::max<size_t>(1, n * out.dpad), st);
    out.sq.alloc(std::max<size_t>(1, n), st);
    out.amax.alloc(1, st);
    QG_CUDA(cudaMemsetAsync(out.amax.get(), 0, sizeof(uint32_t), st));
    if (n == 0) return;
    k_tile_amax<<<std::min(blocks_of(n * dim, 4096), static_cast<unsigned>(8 * sm_count())), 256, 0, st>>>(
        rows, n * dim, out.amax.get());
    QG_LAUNCH_CHECK();
    k_tile_base<<<blocks_of(n * 32), 256, 0, st>>>(rows, n, dim, out.dpad, out.amax.get(),
                                                   reinterpret_cast<__half*>(out.f16.get()), out.sq.get());
    QG_LAUNCH_CHECK();
}

void tile_store(const TileQueries& qs, const uint16_t* base_f16, size_t n, int dpad, float* store, size_t ld, int* err,
                bool may_tune, cudaStream_t st) {
    if (qs.n == 0 || n == 0) return;
    TileArgs a{};
    a.nq = static_cast<int>(qs.n);
    a.kblocks = (dpad + KA - 1) / KA;
    a.ksteps = (qs.dim + 15) / 16;
    a.mtiles = static_cast<int>(ceil_div(qs.n, BM));
    a.ntiles = static_cast<int>(ceil_div(n, BN));
    a.group_n = 16;
    a.err = err;
    a.store = store;
    a.ld = ld;
    a.ncols = static_cast<int>(n);
    const CUtensorMap tmA = make_map(qs.f16.get(), qs.n, qs.dpad, BM);
    const CUtensorMap tmB = make_map(base_f16, n, dpad, BN);
    launch_tile<kStore>(tmA, tmB, a, st, may_tune, [] {}, [] {});
}

// The CTAs that may share a query tile of a nearest launch over ntiles base tiles.
// Each of them appends records of its own: two warps' running minima over 2 ntiles / ctas
// runs of 32 rows each set about ln(2 ntiles / ctas) + 0.6 records, and 256 fit a query's list. (64 to 512
// queries against 16,384 rows spread over 74 to 128 CTAs a tile all overflowed:
// adding 512 x 128 took 1.13 ms, on the exact tiles alone 1.01, and takes 0.62.)
int nearest_ctas(int ntiles) {
    int c = std::min(ntiles, 128);
    while (c > 1 && 2 * c * (std::log(2.0 * ntiles / c) + 0.6) > 0.75 * kNearestCap) --c;
    return c;
}

// One launch over every base row per block of queries: a lane of the epilogue
// owns one query, keeps its smallest upper bound so far and appends the rows
// whose lower bound is at most that. Rows in random order give about ln(n)
// records a query and warp; only those within the bound of the final one are
// scored exactly.
size_t tile_nearest(const float* q, const TileQueries& qs, const float* base_rows, const TileBase& base,
                    uint32_t* label, DevBuf<uint32_t>& redo, cudaStream_t st) {
    const size_t nq = qs.n, n = base.n;
    const int d = base.dim;
    if (nq == 0) return 0;
    require(n >= 1 && n < (size_t{1} << 31) && nq < (size_t{1} << 31), "too many rows for the tensor-core path",
            kUnsupported);
    const TileBound bound(d, false);
    const size_t npad = ceil_div(n, BN) * BN;
    DevBuf<float> xterm(npad, st), run_slack(npad / 32, st);
    k_tile_terms<<<blocks_of(npad), 256, 0, st>>>(base.sq.get(), n, npad, bound, nullptr, nullptr,
                                                   xterm.get(), run_slack.get(), 1, 0, false, nullptr, nullptr);
    QG_LAUNCH_CHECK();
    const size_t QB = 131072;   // queries per block: 268 MB of candidate lists
    const size_t qb = std::min(QB, nq);
    DevBuf<float> qmul(qb, st), qslack(qb, st);
    DevBuf<uint32_t> thr(qb, st), count(qb, st);
    DevBuf<uint2> cand(qb * kNearestCap, st);
    redo.alloc(nq + 2, st);   // the list, its length, and the error flag
    uint32_t* const nredo = redo.get() + nq;
    QG_CUDA(cudaMemsetAsync(nredo, 0, 2 * sizeof(uint32_t), st));
    TileArgs a{};
    a.kblocks = (base.dpad + KA - 1) / KA;
    a.ksteps = (d + 15) / 16;
    a.ntiles = static_cast<int>(ceil_div(n, BN));
    // a base that stays in L2 is walked whole for each query tile, so that the
    // running bound meets every row; a larger one in groups
    // (a quarter of it, at most 16 tiles, for the bound alone, before any row is
    // appended: without it every query's first runs append)
    const bool whole = n * base.dpad * 2 <= (size_t{32} << 20);
    a.group_n = whole ? a.ntiles : 16;
    a.scout = whole ? std::min((a.ntiles + 3) / 4, 16) : 0;
    a.xterm = xterm.get();
    a.run_slack = run_slack.get();
    a.qmul = qmul.get();
    a.qslack = qslack.get();
    a.thr_key = thr.get();
    a.cand_count = count.get();
    a.cand = cand.get();
    a.cap = kNearestCap;
    a.err = reinterpret_cast<int*>(nredo + 1);
    const CUtensorMap tmB = make_map(base.f16.get(), n, base.dpad, BN);
    const bool g4 = (d & 1) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(base_rows) & 7) == 0;
    for (size_t q0 = 0; q0 < nq; q0 += QB) {
        const int nb = static_cast<int>(std::min(QB, nq - q0));
        a.nq = nb;
        a.mtiles = static_cast<int>(ceil_div(static_cast<size_t>(nb), BM));
        a.ctas = std::min(a.mtiles, sm_count()) * nearest_ctas(a.ntiles);
        auto open = [&] {
            k_tile_open<<<blocks_of(nb), 256, 0, st>>>(qs.sq.get() + q0, qs.exps.get() + q0, nb, bound, base.amax.get(),
                                                       kNearestCap, qmul.get(), qslack.get(), thr.get(), count.get());
            QG_LAUNCH_CHECK();
        };
        open();
        const CUtensorMap tmA = make_map(qs.f16.get() + q0 * qs.dpad, nb, qs.dpad, BM);
        {
            KernelTimer kt("mm_filter", st);
            launch_tile<kNearest>(tmA, tmB, a, st, /*may_tune=*/true, [] {}, open);
        }
        const unsigned blocks = blocks_of(nb, 8);
        if (g4)
            k_tile_pick<4><<<blocks, 256, 0, st>>>(q + q0 * d, d, base_rows, nb, count.get(), cand.get(), kNearestCap,
                                                   thr.get(), static_cast<uint32_t>(q0), label + q0, redo.get(), nredo);
        else
            k_tile_pick<8><<<blocks, 256, 0, st>>>(q + q0 * d, d, base_rows, nb, count.get(), cand.get(), kNearestCap,
                                                   thr.get(), static_cast<uint32_t>(q0), label + q0, redo.get(), nredo);
        QG_LAUNCH_CHECK();
    }
    uint32_t h[2] = {0, 0};
    QG_CUDA(cudaMemcpyAsync(h, nredo, sizeof(h), cudaMemcpyDeviceToHost, st));
    QG_CUDA(cudaStreamSynchronize(st));
    require(h[1] == 0, "tensor-core filter: a pipeline wait timed out", kRuntimeError);
    return h[0];
}

// The exact k nearest rows of each query (see "the k nearest" above). sweep: every
// row under one threshold, again with a lower one while a list overflows, for
// queries whose lists overflowed when chunks of growing size were taken: rows stored in
// an order (by cluster, by time) bring what is near all at once, and the threshold
// of the rows before them lets all of it pass.
TileRedo tile_topk(const float* q, const TileQueries& qs, const float* base_rows, const TileBase& base, bool ip, size_t k,
                 const uint64_t* allow, const uint64_t* deny, uint64_t* out_key, uint32_t* out_slot,
                 DevBuf<uint32_t>& redo, bool sweep, cudaStream_t st) {
    const size_t nq = qs.n, n = base.n;
    const int d = base.dim;
    if (nq == 0 || k == 0) return {};
    require(n >= 1 && n < (size_t{1} << 31) && nq < (size_t{1} << 31), "too many rows for the tensor-core path",
            kUnsupported);
    require(k <= kTileMaxK, "k too large for the tensor-core path", kUnsupported);
    // the candidate list: about 8 times what is wanted, so that a chunk of rows
    // far from their average order does not overflow it
    // (few queries take the most there is: rows stored in an order overflow it less)
    const int cap = sweep || nq <= 64 ? kMaxCap : std::clamp(next_pow2(static_cast<int>(8 * k)), 2048, kMaxCap);
    // the sample: enough rows that the first chunk's threshold lets few pass
    const size_t seed = std::min<size_t>(n, std::clamp<size_t>(ceil_div(16 * k, BN) * BN, 2048, 8192));
    const size_t step = n / seed;
    const TileBound bound(d, ip);
    const size_t npad = ceil_div(n, BN) * BN;
    DevBuf<float> xterm(npad, st), run_slack(npad / 32, st), sample_term(seed, st), sample_sq(seed, st);
    k_tile_terms<<<blocks_of(npad), 256, 0, st>>>(base.sq.get(), n, npad, bound, allow, deny, xterm.get(),
                                                   run_slack.get(), static_cast<uint32_t>(step),
                                                   static_cast<uint32_t>(seed), !sweep, sample_term.get(),
                                                   sample_sq.get());
    QG_LAUNCH_CHECK();
    const size_t ld = ceil_div(seed, 4) * 4;
    // queries per block: the lists within 512 MB, the stored products within 256 MB
    const size_t QB = std::min<size_t>({(size_t{512} << 20) / (cap * 8), (size_t{256} << 20) / (ld * 4), nq});
    DevBuf<float> acc(QB * ld, st), qmul(QB, st), qslack(QB, st);
    DevBuf<uint32_t> thr(QB, st), count(QB, st);
    DevBuf<uint2> cand(QB * cap, st);
    // the lists from both ends, their lengths, the error flag, and a sweep's count of lists opened again
    redo.alloc(nq + 4, st);
    uint32_t* const nredo = redo.get() + nq;
    QG_CUDA(cudaMemsetAsync(nredo, 0, 3 * sizeof(uint32_t), st));
    TileArgs a{};
    a.kblocks = (base.dpad + KA - 1) / KA;
    a.ksteps = (d + 15) / 16;
    a.xterm = xterm.get();
    a.run_slack = run_slack.get();
    a.qmul = qmul.get();
    a.qslack = qslack.get();
    a.thr_key = thr.get();
    a.cand_count = count.get();
    a.cand = cand.get();
    a.cap = cap;
    a.err = reinterpret_cast<int*>(nredo + 2);
    a.store = acc.get();
    a.ld = ld;
    const CUtensorMap tmB = make_map(base.f16.get(), n, base.dpad, BN);
    const CUtensorMap tmS = make_map(base.f16.get(), seed, base.dpad, BN, step);
    const size_t seed_smem = seed * 8, cut_smem = static_cast<size_t>(cap) * 12;
    allow_large_smem<k_tile_seed>();
    allow_large_smem<k_tile_cut>();
    allow_large_smem<k_tile_sweep_cut>();
    allow_large_smem<k_tile_finish<4>>();
    allow_large_smem<k_tile_finish<8>>();
    const bool g4 = (d & 1) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(base_rows) & 7) == 0;
    // chunks grow so that about 320 rows pass in each, of a list of at least
    // 2,048 (10,000 queries against 2M x 96, k = 100: the chunks and cuts of
    // growth 3, 4 and 6 took 6.35, 6.32 and 6.52 ms)
    // Up to 8 times at small k (1M x 96, k = 10, growth 4 / 8 / 16 / 32: 65 queries 242 / 207 / 218 /
    // 229 us, 1,000 queries 480 / 456 / 469 / 466, 10,000 queries 3,052 / 2,997 / 3,122 / 3,204), and 32
    // for few queries, whose chunks are short of work (one query 232 / 204 / 200 / 190 us, 16
    // queries 239 / 214 / 219 / 206; at 64 the two are even: 224 and 227).
    const size_t growth = std::clamp<size_t>(1 + 320 / k, 2, nq <= 64 ? 32 : 8);
    for (size_t q0 = 0; q0 < nq; q0 += QB) {
        const int nb = static_cast<int>(std::min(QB, nq - q0));
        a.nq = nb;
        a.mtiles = static_cast<int>(ceil_div(static_cast<size_t>(nb), BM));
        k_tile_open<<<blocks_of(nb), 256, 0, st>>>(qs.sq.get() + q0, qs.exps.get() + q0, nb, bound, base.amax.get(), cap,
                                                   qmul.get(), qslack.get(), thr.get(), count.get());
        QG_LAUNCH_CHECK();
        const CUtensorMap tmA = make_map(qs.f16.get() + q0 * qs.dpad, nb, qs.dpad, BM);
        a.n0 = 0;
        a.ncols = static_cast<int>(seed);
        a.ntiles = static_cast<int>(ceil_div(seed, BN));
        a.group_n = a.ntiles;
        {
            KernelTimer kt("mm_filter", st);
            launch_tile<kStore>(tmA, tmS, a, st, /*may_tune=*/false, [] {}, [] {});
        }
        k_tile_seed<<<nb, 256, seed_smem, st>>>(acc.get(), ld, static_cast<int>(seed), sample_term.get(), sample_sq.get(),
                                                bound.c2, qmul.get(), qslack.get(), static_cast<int>(k), cap,
                                                sweep ? 0u : static_cast<uint32_t>(step), thr.get(), count.get(), cand.get());
        QG_LAUNCH_CHECK();
        for (int left = kSweeps; sweep && left > 0; --left) {
            for (size_t n0 = 0; n0 < n; n0 += kMaxChunkRows) {
                a.n0 = static_cast<int>(n0);
                a.ntiles = static_cast<int>(ceil_div(std::min(n - n0, kMaxChunkRows), BN));
                a.group_n = 16;
                KernelTimer kt("mm_filter", st);
                launch_tile<kFilter>(tmA, tmB, a, st, /*may_tune=*/false, [] {}, [] {});
            }
            uint32_t open = 0;
            QG_CUDA(cudaMemsetAsync(nredo + 3, 0, sizeof(uint32_t), st));
            k_tile_sweep_cut<<<nb, 128, cut_smem, st>>>(base.sq.get(), bound.c2, qslack.get(), static_cast<int>(k), cap,
                                                        left == 1, thr.get(), count.get(), cand.get(), nredo + 3);
            QG_LAUNCH_CHECK();
            QG_CUDA(cudaMemcpyAsync(&open, nredo + 3, sizeof(open), cudaMemcpyDeviceToHost, st));
            QG_CUDA(cudaStreamSynchronize(st));
            if (open == 0) break;
        }
        for (size_t n0 = sweep || seed == n ? n : 0; n0 < n;) {
            const size_t n1 = std::min({n, (n0 + seed) * growth - seed, n0 + kMaxChunkRows});   // (the sample counts)
            a.n0 = static_cast<int>(n0);
            a.ntiles = static_cast<int>(ceil_div(n1 - n0, BN));
            a.group_n = 16;
            {
                KernelTimer kt("mm_filter", st);
                // (a timed run's appends go over those of the run before it)
                DevBuf<uint32_t> before;
                launch_tile<kFilter>(
                    tmA, tmB, a, st, /*may_tune=*/true,
                    [&] {
                        before.alloc(nb, st);
                        QG_CUDA(cudaMemcpyAsync(before.get(), count.get(), nb * 4, cudaMemcpyDeviceToDevice, st));
                    },
                    [&] { QG_CUDA(cudaMemcpyAsync(count.get(), before.get(), nb * 4, cudaMemcpyDeviceToDevice, st)); });
            }
            n0 = n1;
            if (n0 == n) break;
            k_tile_cut<<<nb, 128, cut_smem, st>>>(base.sq.get(), bound.c2, qslack.get(), static_cast<int>(k), cap,
                                                  thr.get(), count.get(), cand.get());
            QG_LAUNCH_CHECK();
        }
        auto finish = [&](auto kernel) {
            kernel<<<nb, 256, cut_smem, st>>>(q + q0 * d, d, base_rows, ip, base.sq.get(), bound.c2, qslack.get(),
                                              static_cast<int>(k), cap, count.get(), thr.get(), cand.get(),
                                              Sample{acc.get(), ld, static_cast<int>(seed), sample_term.get(),
                                                     sample_sq.get()},
                                              qmul.get(), static_cast<uint32_t>(q0), out_key + q0 * k, out_slot + q0 * k, redo.get(),
                                              static_cast<uint32_t>(nq), nredo);
            QG_LAUNCH_CHECK();
        };
        if (g4) finish(k_tile_finish<4>);
        else finish(k_tile_finish<8>);
    }
    uint32_t h[3] = {0, 0, 0};
    QG_CUDA(cudaMemcpyAsync(h, nredo, sizeof(h), cudaMemcpyDeviceToHost, st));
    QG_CUDA(cudaStreamSynchronize(st));
    require(h[2] == 0, "tensor-core filter: a pipeline wait timed out", kRuntimeError);
    return {h[0], h[1]};
}

} // namespace qg
