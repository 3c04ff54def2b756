// Coarse assignment through the tensor cores (reference src/ivf_index.cpp:
// 305-419, which ranks lists by the exact distance, ties by list). The tile
// engine's store mode gives acc(q, c), the F16 dot product of a query and a
// centroid (each row scaled by a power of two first, undone exactly after)
// accumulated in FP32. With e = C (|q|^2 + |c|^2) (C and its terms: the top of
// qg_tile.cu), each exact score lies in [lb, ub] = [s^ - e, s^ + e] (s^ =
// |q|^2 + |c|^2 - 2 acc for L2, -acc for inner product, e halved). T, the P-th
// smallest ub, bounds the P-th exact score from above, so only centroids with
// lb <= T can be among the P nearest: k_coarse_recheck scores those exactly,
// in the reference's order, and keeps the P smallest by (score, list), -0 == +0.
#include "qg_device.cuh"
#include "qg_ops.h"
#include "qg_search.h"
#include "qg_tile.h"

#include <algorithm>
#include <cmath>

namespace qg {

// x * 2^e rounded to nearest, which is what ldexpf returns: one multiply by
// 2^e when that is a normal float (the product is then the correctly rounded
// x * 2^e), ldexpf itself otherwise.
__device__ __forceinline__ float scale_pow2(float x, int e) {
    return (e >= -126 && e <= 127) ? __fmul_rn(x, __int_as_float((e + 127) << 23)) : ldexpf(x, e);
}

// The P smallest of the cnt distinct keys key[0, cnt) written in order, key by
// key, for P <= cnt <= 32 K x warps: each warp sorts a run of up to 32 K keys
// in registers; a key's rank is then the number of keys below it in each run
// (binary searches over the sorted runs; its own run counts its place in it),
// and a key of rank < P goes to place rank. One block barrier.
template <int K>
__device__ void ranked_out(uint64_t* key, int cnt, int P, const float* score_of, uint32_t* probe_q, float* pdist_q) {
    constexpr int R = 32 * K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int n_w = max(0, min(R, cnt - R * warp));
    if (n_w > 0) warp_sort_keys_reg<K>(key + R * warp, n_w);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int e = R * warp + i * 32 + lane;
        if (e >= cnt) continue;
        const uint64_t k = key[e];
        int rank = 0;
        for (int w = 0; w < nw; ++w) {
            const int len = max(0, min(R, cnt - R * w));
            const uint64_t* run = key + R * w;
            int pos = 0;   // keys of the run below k
#pragma unroll
            for (int step = R; step > 0; step >>= 1)
                if (pos + step <= len && run[pos + step - 1] < k) pos += step;
            rank += pos;
        }
        if (rank < P) {
            const uint32_t j = static_cast<uint32_t>(k);
            probe_q[rank] = j;
            pdist_q[rank] = score_of[j];
        }
    }
}

// What the recheck of one query reads and writes.
struct RecheckArgs {
    const float *q, *q2;
    const int* qexp;
    const float *cent, *c2;
    const int* cexp;
    int nlist, d;
    bool ip;
    float c_up, c_lo;
    const float* accm;
    size_t ld;
    int P;
    uint32_t* probe;
    float* pdist;
    uint32_t *list, *nlist_redo;   // queries left to k_coarse_redo, and how many
    int* nredone;                  // statistics: those queries,
    unsigned long long* ncand;     // and the lists rescored exactly
};

// One query by one block, with room for cap candidates. can_defer: a query of
// extreme norm, or with more candidates than that (too many near-ties), goes on
// the list instead; otherwise cap holds every list.
__device__ __forceinline__ void recheck_query(const RecheckArgs& ra, int qi, int cap, bool can_defer) {
    extern __shared__ __align__(16) uint8_t sm_raw[];
    const float *q = ra.q, *q2 = ra.q2, *cent = ra.cent, *c2 = ra.c2, *accm = ra.accm;
    const int *qexp = ra.qexp, *cexp = ra.cexp;
    const int nlist = ra.nlist, d = ra.d, P = ra.P;
    const bool ip = ra.ip;
    const float c_up = ra.c_up, c_lo = ra.c_lo;
    const size_t ld = ra.ld;
    uint32_t* const probe = ra.probe;
    float* const pdist = ra.pdist;
    auto defer = [&] {
        if (threadIdx.x == 0) {
            ra.list[atomicAdd(ra.nlist_redo, 1u)] = static_cast<uint32_t>(qi);
            atomicAdd(ra.nredone, 1);
        }
    };
    uint64_t* ckey = reinterpret_cast<uint64_t*>(sm_raw);             // cap
    float* qv = reinterpret_cast<float*>(ckey + cap);                   // d, 16-byte aligned
    uint32_t* ub = reinterpret_cast<uint32_t*>(qv + ((d + 3) & ~3));    // nlist
    __shared__ int hist[kKeyHist], s_count, s_wfin[8];
    __shared__ uint32_t s_wmin[8], s_wmax[8], s_t;
    const float* arow = accm + static_cast<size_t>(qi) * ld;
    const float qq = q2[qi];
    const int qe = qexp[qi];
    // norms where float squares lose relative accuracy (underflow or near
    // overflow): the relative bound does not hold, so such a query takes the
    // exact path and such a list is always rescored
    auto extreme = [](float x2) { return (x2 > 0.0f && x2 < 0x1p-60f) || !(x2 < 0x1p60f); };
    const bool all = extreme(qq);   // every list rescored
    if (all && can_defer) {
        defer();
        return;
    }
    for (int t = threadIdx.x; t < d; t += blockDim.x) qv[t] = q[static_cast<size_t>(qi) * d + t];
    for (int t = threadIdx.x; t < kKeyHist; t += blockDim.x) hist[t] = 0;
    // upper bounds, rounded up at every step (c_up >= 1 + C for L2, >= C / 2
    // for inner product; the f16 row scaling is undone exactly by scale_pow2).
    // Four lists per thread and step, read as 16-byte vectors.
    auto upper = [&](float acc_j, float c2j, int cej) -> uint32_t {
        const float s = __fadd_ru(qq, c2j);
        const float a = scale_pow2(acc_j, -(qe + cej));
        const float hi = ip ? __fmaf_ru(c_up, s, -a) : __fmaf_ru(-2.0f, a, __fmul_ru(c_up, s));
        return extreme(c2j) ? 0xFFFFFFFFu : float_key(hi);
    };
    // (and the range and count of the bounded ones, for the threshold)
    uint32_t kmin = 0xFFFFFFFFu, kmax = 0;
    int nfin = 0;
    auto keep = [&](int j, uint32_t u) {
        ub[j] = u;
        if (u != 0xFFFFFFFFu) {
            kmin = min(kmin, u);
            kmax = max(kmax, u);
            ++nfin;
        }
    };
    const int n4 = nlist & ~3;
    for (int j = 4 * threadIdx.x; j < n4; j += 4 * blockDim.x) {
        const float4 av = *reinterpret_cast<const float4*>(arow + j);
        const float4 cv = *reinterpret_cast<const float4*>(c2 + j);
        const int4 ev = *reinterpret_cast<const int4*>(cexp + j);
        keep(j, upper(av.x, cv.x, ev.x));
        keep(j + 1, upper(av.y, cv.y, ev.y));
        keep(j + 2, upper(av.z, cv.z, ev.z));
        keep(j + 3, upper(av.w, cv.w, ev.w));
    }
    for (int j = n4 + threadIdx.x; j < nlist; j += blockDim.x) keep(j, upper(arow[j], c2[j], cexp[j]));
    for (int o = 16; o > 0; o >>= 1) {
        kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
        kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        nfin += __shfl_xor_sync(0xffffffffu, nfin, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_wmin[threadIdx.x >> 5] = kmin;
        s_wmax[threadIdx.x >> 5] = kmax;
        s_wfin[threadIdx.x >> 5] = nfin;
    }
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (int w = 0; w < 8; ++w) {
        kmin = min(kmin, s_wmin[w]);
        kmax = max(kmax, s_wmax[w]);
    }
    nfin = 0;
    for (int w = 0; w < 8; ++w) nfin += s_wfin[w];
    const uint32_t T = block_threshold_u32(ub, nlist, P, kmin, kmax, nfin, hist, &s_t);
    // candidates: lower bound, rounded down (c_lo <= 1 - C for L2; for inner
    // product the margin c_up is subtracted from a sum rounded up), <= T
    auto lower_in = [&](float acc_j, float c2j, int cej) -> bool {
        const float a = scale_pow2(acc_j, -(qe + cej));
        const float lo = ip ? __fmaf_rd(-c_up, __fadd_ru(qq, c2j), -a)
                            : __fmaf_rd(-2.0f, a, __fmul_rd(c_lo, __fadd_rd(qq, c2j)));
        return all || float_key(lo) <= T || extreme(c2j);
    };
    auto push = [&](int j) {
        const int pos = atomicAdd(&s_count, 1);
        if (pos < cap) ckey[pos] = static_cast<uint64_t>(j);
    };
    for (int j = 4 * threadIdx.x; j < n4; j += 4 * blockDim.x) {
        const float4 av = *reinterpret_cast<const float4*>(arow + j);
        const float4 cv = *reinterpret_cast<const float4*>(c2 + j);
        const int4 ev = *reinterpret_cast<const int4*>(cexp + j);
        if (lower_in(av.x, cv.x, ev.x)) push(j);
        if (lower_in(av.y, cv.y, ev.y)) push(j + 1);
        if (lower_in(av.z, cv.z, ev.z)) push(j + 2);
        if (lower_in(av.w, cv.w, ev.w)) push(j + 3);
    }
    for (int j = n4 + threadIdx.x; j < nlist; j += blockDim.x)
        if (lower_in(arow[j], c2[j], cexp[j])) push(j);
    __syncthreads();
    const int cnt = s_count;
    if (cnt > cap) {   // (cap >= nlist when it cannot be deferred)
        if (can_defer) defer();
        return;
    }
    if (threadIdx.x == 0) atomicAdd(ra.ncand, static_cast<unsigned long long>(cnt));
    // exact scores, one candidate per 8-lane group; each list's score is kept
    // by list (over its upper bound, no longer needed) for the output
    float* score_of = reinterpret_cast<float*>(ub);
    if ((d & 1) == 0 && (reinterpret_cast<uintptr_t>(cent) & 7) == 0) {
        // rows 8-byte aligned: one candidate per 4-lane group, one 32-byte
        // sector of its row per step
        const int ngrp = blockDim.x >> 2, grp = threadIdx.x >> 2;
        const int rounds = (cnt + ngrp - 1) / ngrp;   // (block-uniform)
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = rd * ngrp + grp;
            const bool act = i < cnt;
            const int j = act ? static_cast<int>(ckey[i]) : 0;   // idle groups score row 0 unused
            const float* row = cent + static_cast<size_t>(j) * d;
            const float sc = ip ? -exact_avx2_group4<false>(qv, row, d) : exact_avx2_group4<true>(qv, row, d);
            if (act && (threadIdx.x & 3) == 0) {
                ckey[i] = (static_cast<uint64_t>(float_key_eq0(sc)) << 32) | static_cast<uint32_t>(j);
                score_of[j] = sc;
            }
        }
    } else {
        const int ngrp = blockDim.x >> 3, grp = threadIdx.x >> 3;
        const int rounds = (cnt + ngrp - 1) / ngrp;   // (block-uniform)
        for (int rd = 0; rd < rounds; ++rd) {
            const int i = rd * ngrp + grp;
            const bool act = i < cnt;
            const int j = act ? static_cast<int>(ckey[i]) : 0;   // idle groups score row 0 unused
            const float* row = cent + static_cast<size_t>(j) * d;
            const float sc = ip ? -exact_avx2_group8<false, true>(qv, row, d) : exact_avx2_group8<true, true>(qv, row, d);
            if (act && (threadIdx.x & 7) == 0) {
                ckey[i] = (static_cast<uint64_t>(float_key_eq0(sc)) << 32) | static_cast<uint32_t>(j);
                score_of[j] = sc;
            }
        }
    }
    __syncthreads();
    // the P smallest by (score, list), in order
    if (cnt <= 32 * (static_cast<int>(blockDim.x) >> 5)) {
        ranked_out<1>(ckey, cnt, P, score_of, probe + static_cast<size_t>(qi) * P, pdist + static_cast<size_t>(qi) * P);
        return;
    }
    if (cnt <= 64 * (static_cast<int>(blockDim.x) >> 5)) {
        ranked_out<2>(ckey, cnt, P, score_of, probe + static_cast<size_t>(qi) * P, pdist + static_cast<size_t>(qi) * P);
        return;
    }
    if (cnt > P) {
        if (threadIdx.x < 32) warp_select_keep(ckey, cnt, P, hist);
        __syncthreads();
    }
    const int ns = next_pow2(P < 2 ? 2 : P);
    for (int i = P + threadIdx.x; i < ns; i += blockDim.x) ckey[i] = ~0ull;
    bitonic_sort_keys(ckey, ns);
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const uint32_t j = static_cast<uint32_t>(ckey[i]);
        probe[static_cast<size_t>(qi) * P + i] = j;
        pdist[static_cast<size_t>(qi) * P + i] = score_of[j];
    }
}

__global__ void __launch_bounds__(256, 6) k_coarse_recheck(RecheckArgs ra, int cap, bool can_defer) {
    recheck_query(ra, blockIdx.x, cap, can_defer);
}

// The queries on the list, with room for every list: a few blocks that take
// one after the other (none, nearly always, so the list is not read back to
// the host to decide; the launch costs 3 us, the read-back cost the search a
// wait of about 30).
__global__ void __launch_bounds__(256) k_coarse_redo(RecheckArgs ra, int cap) {
    const uint32_t n = *ra.nlist_redo;
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {   // (block-uniform)
        recheck_query(ra, static_cast<int>(ra.list[i]), cap, false);
        __syncthreads();
    }
}

static size_t coarse_recheck_smem(int nlist, int d, int cap) {
    return static_cast<size_t>(cap) * 8 + static_cast<size_t>((d + 3) & ~3) * 4 + static_cast<size_t>(nlist) * 4;
}

static int coarse_cap(int nlist, int P) {
    return std::min(next_pow2(nlist), std::max(1024, next_pow2(4 * P)));
}

bool coarse_mm_supported(int nlist, int dim, int P, bool cent_prepared) {
    const int cap = next_pow2(nlist);
    return cent_prepared && tile_supported(dim) && P >= 1 && P <= nlist && nlist <= 16384 &&
           coarse_recheck_smem(nlist, dim, cap) <= 200 * 1024;
}

void coarse_probes_mm(const IvfView& v, const float* q, int nq, int P, uint32_t* probe, float* pdist, int* flags,
                      bool hold_all, bool may_tune, cudaStream_t st) {
    if (nq == 0) return;
    const int d = v.dim, nlist = v.nlist;
    allow_large_smem<k_coarse_recheck>();
    allow_large_smem<k_coarse_redo>();
    const size_t QB = 65536;   // query blocks bound the score matrix
    for (size_t q0 = 0; q0 < static_cast<size_t>(nq); q0 += QB) {
        const int nb = static_cast<int>(std::min(QB, static_cast<size_t>(nq) - q0));
        TileQueries qs;
        tile_prepare_queries(q + q0 * d, nb, d, qs, st);
        const size_t ld = (static_cast<size_t>(nlist) + 3) & ~size_t{3};
        DevBuf<float> accm(static_cast<size_t>(nb) * ld, st);
        {
            KernelTimer kt("coarse_mm", st);
            tile_store(qs, v.cent_f16, nlist, v.cent_dpad, accm.get(), ld, flags + 2, may_tune, st);
        }
        const double C = tile_error_factor(d);
        RecheckArgs ra{};
        ra.q = q + q0 * d;
        ra.q2 = qs.sq.get();
        ra.qexp = qs.exps.get();
        ra.cent = v.centroids;
        ra.c2 = v.cent_sq;
        ra.cexp = v.cent_exp;
        ra.nlist = nlist;
        ra.d = d;
        ra.ip = v.ip_metric;
        // the bound's factors as floats rounded outwards
        ra.c_up = v.ip_metric ? std::nextafter(static_cast<float>(0.5 * C), 1.0f)
                              : std::nextafter(static_cast<float>(1.0 + C), 2.0f);
        ra.c_lo = std::nextafter(static_cast<float>(1.0 - C), 0.0f);
        ra.accm = accm.get();
        ra.ld = ld;
        ra.P = P;
        ra.probe = probe + q0 * P;
        ra.pdist = pdist + q0 * P;
        ra.nredone = flags + 3;
        ra.ncand = reinterpret_cast<unsigned long long*>(flags + 4);
        const int full = next_pow2(nlist);
        const int cap = hold_all ? full : coarse_cap(nlist, P);
        const bool defer = cap < full;
        DevBuf<uint32_t> list;
        if (defer) {
            list.alloc(static_cast<size_t>(nb) + 1, st);
            ra.list = list.get();
            ra.nlist_redo = list.get() + nb;
            QG_CUDA(cudaMemsetAsync(ra.nlist_redo, 0, sizeof(uint32_t), st));
        }
        KernelTimer kt("coarse_recheck", st);
        k_coarse_recheck<<<static_cast<unsigned>(nb), 256, coarse_recheck_smem(nlist, d, cap), st>>>(ra, cap, defer);
        QG_LAUNCH_CHECK();
        if (defer) {
            k_coarse_redo<<<static_cast<unsigned>(std::min(nb, 148)), 256, coarse_recheck_smem(nlist, d, full), st>>>(
                ra, full);
            QG_LAUNCH_CHECK();
        }
    }
}

} // namespace qg
