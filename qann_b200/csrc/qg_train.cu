// Device steps of training: assignment for small codebooks, member sums in
// point order, distances to the own centroid, and row gathers. The host side
// (qg_train_host.cpp) replays the reference's random choices and bookkeeping
// around them.
#include "qg_device.cuh"
#include "qg_ops.h"
#include "qg_train.h"

namespace qg {

// thread per (problem, point): k exact distances, first index of the minimum
// (the reference's nearest_centroid keeps the first strictly smaller one;
// reference src/kmeans.cpp:102-115)
__global__ void k_assign_small(const float* __restrict__ x, size_t n, int d, const float* __restrict__ c, int k, int P,
                               uint32_t* __restrict__ assign) {
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * P) return;
    const size_t p = t / n;
    const float* pt = x + t * d;
    const float* cp = c + p * static_cast<size_t>(k) * d;
    float best = 3.402823466e+38f;   // FLT_MAX, the reference's starting value
    uint32_t bi = 0;
    for (int j = 0; j < k; ++j) {
        const float dist = exact_avx2<true>(pt, cp + static_cast<size_t>(j) * d, d);
        if (dist < best) {
            best = dist;
            bi = static_cast<uint32_t>(j);
        }
    }
    assign[t] = bi;
}

void assign_small(const float* x, size_t n, int d, const float* c, int k, int P, uint32_t* assign, cudaStream_t st) {
    if (n == 0) return;
    k_assign_small<<<static_cast<unsigned>(ceil_div(n * P, 128)), 128, 0, st>>>(x, n, d, c, k, P, assign);
    QG_LAUNCH_CHECK();
}

// Member sums: float sums over a centroid's members in the order given, one
// after the other, so the members' loads are what can overlap. A warp per
// (problem, centroid, 32 dims): the lanes fetch 32 member indices at once, the
// next 32 under the work on these, and 8 members' rows are in flight ahead of the
// adds. (A thread per sum waited for an index and then a row every few members:
// 187 us for 500,000 x 128 in 4,096 clusters, 129 now.)
__global__ void __launch_bounds__(256) k_member_sums(const float* __restrict__ x, size_t n, int d,
                                                     const uint32_t* __restrict__ order,
                                                     const uint32_t* __restrict__ off, int k, int P,
                                                     float* __restrict__ out) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, parts = (d + 31) / 32;
    const size_t w = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (w >= static_cast<size_t>(P) * k * parts) return;
    const size_t pc = w / parts;
    const int l = static_cast<int>(w % parts) * 32 + lane;
    const size_t p = pc / k;
    const int c = static_cast<int>(pc % k);
    const uint32_t* o = order + p * n;
    const uint32_t* f = off + p * (k + 1);
    const float* xp = x + p * n * d + min(l, d - 1);   // (lanes past the last dim read it, unused)
    const uint32_t end = f[c + 1];
    uint32_t i = f[c];
    uint32_t next = i + lane < end ? o[i + lane] : 0u;
    float s = 0.0f;
    for (; i < end; i += 32) {
        const uint32_t mine = next;
        next = i + 32 + lane < end ? o[i + 32 + lane] : 0u;
        const int cnt = static_cast<int>(min(32u, end - i));
        for (int j = 0; j < cnt; j += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)   // (past the last member: row 0, unused)
                v[u] = xp[static_cast<size_t>(__shfl_sync(kFull, mine, j + u)) * d];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < cnt) s = __fadd_rn(s, v[u]);
        }
    }
    if (l < d) out[pc * d + l] = s;
}

// For few dims (PQ sub-spaces): a warp per (problem, centroid), a member per
// lane; its values go round by shuffles, and every lane adds them in order (64
// problems of 4,096 points x 2 dims in 16 clusters: 59 -> 21 us).
template <int D>
__global__ void __launch_bounds__(256) k_member_sums_narrow(const float* __restrict__ x, size_t n,
                                                            const uint32_t* __restrict__ order,
                                                            const uint32_t* __restrict__ off, int k, int P,
                                                            float* __restrict__ out) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const size_t pc = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (pc >= static_cast<size_t>(P) * k) return;
    const size_t p = pc / k;
    const int c = static_cast<int>(pc % k);
    const uint32_t* o = order + p * n;
    const uint32_t* f = off + p * (k + 1);
    const float* xp = x + p * n * D;
    const uint32_t end = f[c + 1];
    uint32_t i = f[c];
    float s[D], next[D];
    auto fetch = [&](uint32_t at) {
        const size_t r = at + lane < end ? o[at + lane] : 0u;
#pragma unroll
        for (int l = 0; l < D; ++l) next[l] = xp[r * D + l];
    };
#pragma unroll
    for (int l = 0; l < D; ++l) s[l] = 0.0f;
    if (i < end) fetch(i);
    for (; i < end; i += 32) {
        float v[D];
#pragma unroll
        for (int l = 0; l < D; ++l) v[l] = next[l];
        if (i + 32 < end) fetch(i + 32);
        const int cnt = static_cast<int>(min(32u, end - i));
        for (int j = 0; j < cnt; ++j)
#pragma unroll
            for (int l = 0; l < D; ++l) s[l] = __fadd_rn(s[l], __shfl_sync(kFull, v[l], j));
    }
#pragma unroll
    for (int l = 0; l < D; ++l)
        if (lane == l) out[pc * D + l] = s[l];
}

void member_sums(const float* x, size_t n, int d, const uint32_t* order, const uint32_t* off, int k, int P, float* out,
                 cudaStream_t st) {
    if (static_cast<size_t>(k) * d * P == 0) return;
    const size_t pc = static_cast<size_t>(k) * P;
    const unsigned narrow = static_cast<unsigned>(ceil_div(pc * 32, 256));
    switch (d) {
        case 1: k_member_sums_narrow<1><<<narrow, 256, 0, st>>>(x, n, order, off, k, P, out); break;
        case 2: k_member_sums_narrow<2><<<narrow, 256, 0, st>>>(x, n, order, off, k, P, out); break;
        case 3: k_member_sums_narrow<3><<<narrow, 256, 0, st>>>(x, n, order, off, k, P, out); break;
        case 4: k_member_sums_narrow<4><<<narrow, 256, 0, st>>>(x, n, order, off, k, P, out); break;
        default:
            k_member_sums<<<static_cast<unsigned>(ceil_div(pc * ((d + 31) / 32) * 32, 256)), 256, 0, st>>>(
                x, n, d, order, off, k, P, out);
    }
    QG_LAUNCH_CHECK();
}

// The same by a 4-lane group per point (even d, 8-byte aligned rows), which
// reads its rows a sector at a time.
__global__ void __launch_bounds__(256) k_own_dist4(const float* __restrict__ x, size_t n, int d,
                                                   const float* __restrict__ c, int k,
                                                   const uint32_t* __restrict__ assign, int P,
                                                   float* __restrict__ dist) {
    const size_t t = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 2;
    const bool in = t < n * P;   // (whole warps call the group scorer together)
    const size_t i = in ? t : 0;
    const float s = exact_avx2_group4<true>(x + i * d, c + (i / n * k + assign[i]) * static_cast<size_t>(d), d);
    if (in && (threadIdx.x & 3) == 0) dist[i] = s;
}

__global__ void k_own_dist(const float* __restrict__ x, size_t n, int d, const float* __restrict__ c, int k,
                           const uint32_t* __restrict__ assign, int P, float* __restrict__ dist) {
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * P) return;
    const size_t p = t / n;
    dist[t] = exact_avx2<true>(x + t * d, c + (p * k + assign[t]) * static_cast<size_t>(d), d);
}

void own_dist(const float* x, size_t n, int d, const float* c, int k, const uint32_t* assign, int P, float* dist,
              cudaStream_t st) {
    if (n == 0) return;
    if ((d & 1) == 0 && (reinterpret_cast<uintptr_t>(x) & 7) == 0 && (reinterpret_cast<uintptr_t>(c) & 7) == 0)
        k_own_dist4<<<static_cast<unsigned>(ceil_div(n * P * 4, 256)), 256, 0, st>>>(x, n, d, c, k, assign, P, dist);
    else
        k_own_dist<<<static_cast<unsigned>(ceil_div(n * P, 128)), 128, 0, st>>>(x, n, d, c, k, assign, P, dist);
    QG_LAUNCH_CHECK();
}

__global__ void k_gather_rows(const float* __restrict__ src, const uint32_t* __restrict__ idx, size_t n, int d,
                              float* __restrict__ out) {
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * d) return;
    const size_t i = t / d;
    out[t] = src[static_cast<size_t>(idx[i]) * d + (t % d)];
}

void gather_rows(const float* src, const uint32_t* idx, size_t n, int d, float* out, cudaStream_t st) {
    if (n == 0) return;
    k_gather_rows<<<static_cast<unsigned>(ceil_div(n * d, 256)), 256, 0, st>>>(src, idx, n, d, out);
    QG_LAUNCH_CHECK();
}

// mean[j] = (double(x[0][j]) + double(x[1][j]) + ...) / n, in row order. One
// thread per column; loads run 8 rows ahead of the dependent adds.
__global__ void k_col_means(const float* __restrict__ x, size_t n, int d, double* __restrict__ mean) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= d) return;
    double s = 0.0;
    size_t i = 0;
    for (; i + 8 <= n; i += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = x[(i + u) * d + j];
#pragma unroll
        for (int u = 0; u < 8; ++u) s = __dadd_rn(s, static_cast<double>(v[u]));
    }
    for (; i < n; ++i) s = __dadd_rn(s, static_cast<double>(x[i * d + j]));
    mean[j] = __ddiv_rn(s, static_cast<double>(n));
}

// cov[t] = sum over rows in order of fma(xc[p], xc[q], cov), xc = double(x) -
// mean, for the pair t = (p, q) = (pairs[t] >> 16, pairs[t] & 0xFFFF). Rows
// are centred into shared memory `tile` rows at a time.
__global__ void __launch_bounds__(256) k_cov_upper(const float* __restrict__ x, size_t n, int d,
                                                   const double* __restrict__ mean, const uint32_t* __restrict__ pairs,
                                                   int npairs, int tile, double* __restrict__ cov) {
    extern __shared__ double xs[];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = t < npairs;
    const int p = live ? static_cast<int>(pairs[t] >> 16) : 0;
    const int q = live ? static_cast<int>(pairs[t] & 0xFFFFu) : 0;
    double acc = 0.0;
    for (size_t i0 = 0; i0 < n; i0 += tile) {
        const int rows = static_cast<int>(n - i0 < static_cast<size_t>(tile) ? n - i0 : tile);
        __syncthreads();
        for (int e = threadIdx.x; e < rows * d; e += blockDim.x) {
            const int j = e % d;
            xs[e] = __dsub_rn(static_cast<double>(x[i0 * d + e]), mean[j]);
        }
        __syncthreads();
        if (live)
            for (int r = 0; r < rows; ++r) acc = __fma_rn(xs[r * d + p], xs[r * d + q], acc);
    }
    if (live) cov[t] = acc;
}

std::vector<double> covariance(const float* x, size_t n, int d, cudaStream_t st) {
    require(n > 0, "training set must not be empty");
    require(d <= 6144, "the GPU rotation training supports dim <= 6144", kUnsupported);
    DevBuf<double> mean(d, st);
    k_col_means<<<static_cast<unsigned>(ceil_div(d, 32)), 32, 0, st>>>(x, n, d, mean.get());
    QG_LAUNCH_CHECK();
    std::vector<uint32_t> pairs;
    pairs.reserve(static_cast<size_t>(d) * (d + 1) / 2);
    for (int p = 0; p < d; ++p)
        for (int q = p; q < d; ++q) pairs.push_back(static_cast<uint32_t>(p) << 16 | static_cast<uint32_t>(q));
    const int np = static_cast<int>(pairs.size());
    DevBuf<uint32_t> dp(np, st);
    QG_CUDA(cudaMemcpyAsync(dp.get(), pairs.data(), np * 4, cudaMemcpyHostToDevice, st));
    DevBuf<double> dc(np, st);
    const int tile = std::max(1, std::min(64, 6144 / d));   // <= 48 KB of centred rows
    k_cov_upper<<<static_cast<unsigned>(ceil_div(np, 256)), 256, static_cast<size_t>(tile) * d * 8, st>>>(
        x, n, d, mean.get(), dp.get(), np, tile, dc.get());
    QG_LAUNCH_CHECK();
    std::vector<double> upper(np);
    QG_CUDA(cudaMemcpyAsync(upper.data(), dc.get(), np * 8, cudaMemcpyDeviceToHost, st));
    QG_CUDA(cudaStreamSynchronize(st));
    const double scale = n > 1 ? 1.0 / static_cast<double>(n - 1) : 1.0;
    std::vector<double> cov(static_cast<size_t>(d) * d);
    for (int t = 0; t < np; ++t) {
        const size_t p = pairs[t] >> 16, q = pairs[t] & 0xFFFFu;
        cov[p * d + q] = upper[t] * scale;
        cov[q * d + p] = cov[p * d + q];
    }
    return cov;
}

__global__ void k_residuals(const float* __restrict__ x, size_t n, int d, const float* __restrict__ centers,
                            const uint32_t* __restrict__ assign, float* __restrict__ out) {
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * d) return;
    const size_t i = t / d;
    out[t] = __fsub_rn(x[t], centers[static_cast<size_t>(assign[i]) * d + (t % d)]);
}

void residuals(const float* x, size_t n, int d, const float* centers, const uint32_t* assign, float* out,
               cudaStream_t st) {
    if (n == 0) return;
    k_residuals<<<static_cast<unsigned>(ceil_div(n * d, 256)), 256, 0, st>>>(x, n, d, centers, assign, out);
    QG_LAUNCH_CHECK();
}

__global__ void k_split_columns(const float* __restrict__ x, size_t n, int dim, int d, int P, float* __restrict__ out) {
    const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * dim) return;
    const size_t i = t / dim;
    const int col = static_cast<int>(t % dim);
    const int p = col / d, l = col % d;
    out[(static_cast<size_t>(p) * n + i) * d + l] = x[t];
}

void split_columns(const float* x, size_t n, int dim, int d, int P, float* out, cudaStream_t st) {
    if (n == 0) return;
    (void)P;
    k_split_columns<<<static_cast<unsigned>(ceil_div(n * dim, 256)), 256, 0, st>>>(x, n, dim, d, P, out);
    QG_LAUNCH_CHECK();
}

} // namespace qg
