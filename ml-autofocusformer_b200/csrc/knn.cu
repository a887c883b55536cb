// k nearest neighbours of 2-D points: for every query the k database points of its batch element at
// the smallest Euclidean distance, ascending, ties towards the lower database index.
//
// This is the neighbourhood search AutoFocusFormer runs before every stage: each token looks for its
// nearest cluster centres (models/aff_transformer.py:476 of the reference, k = 6 of at most 1152
// centres) and, in the adaptive downsampling, for its nearest other token (:298, k = 2).  The reference
// evaluates it with a pykeops LazyTensor reduction (models/point_utils.py:27-58).  Here a thread owns a
// query and keeps its k best candidates in registers while the CTA streams the database through shared
// memory; distances are exact fp32 (sqrt(dx*dx + dy*dy)), no matrix-multiply shortcut.
#include <math_constants.h>

#include "common.cuh"

namespace clusten {
namespace {

constexpr int kKnnThreads = 128;
constexpr int kKnnTile = 2048;          // database points staged at a time (16 KB)

// squared distances to two points
__device__ __forceinline__ float2 dist2(float qx, float qy, const float4& p) {
    const float dx0 = qx - p.x, dy0 = qy - p.y, dx1 = qx - p.z, dy1 = qy - p.w;
    return make_float2(dx0 * dx0 + dy0 * dy0, dx1 * dx1 + dy1 * dy1);
}

template <int K>
__global__ void __launch_bounds__(kKnnThreads)
knn2d_kernel(const float2* __restrict__ query, const float2* __restrict__ db, int nq, int n,
             int64_t* __restrict__ idx_out, float* __restrict__ dist_out) {
    __shared__ __align__(16) float2 pts[kKnnTile + 4];
    const int b = blockIdx.y;
    const int qi = blockIdx.x * kKnnThreads + threadIdx.x;
    const bool live = qi < nq;
    const float2 q = live ? query[(long long)b * nq + qi] : make_float2(0.f, 0.f);
    const float2* dbb = db + (long long)b * n;
    float best[K];
    int who[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
        best[i] = CUDART_INF_F;
        who[i] = 0x7fffffff;
    }
    // in order of (distance, index): whatever order the points come in, the result is the same
    auto insert = [&](float d, int w) {
        bool before[K];
#pragma unroll
        for (int s = 0; s < K; ++s) before[s] = d < best[s] || (d == best[s] && w < who[s]);
#pragma unroll
        for (int s = K - 1; s > 0; --s) {
            best[s] = before[s] ? (before[s - 1] ? best[s - 1] : d) : best[s];
            who[s] = before[s] ? (before[s - 1] ? who[s - 1] : w) : who[s];
        }
        best[0] = before[0] ? d : best[0];
        who[0] = before[0] ? w : who[0];
    };
    for (int t0 = 0; t0 < n; t0 += kKnnTile) {
        const int cnt = min(kKnnTile, n - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += kKnnThreads) pts[i] = dbb[t0 + i];
        // filled up to a multiple of four points
        if (threadIdx.x < 4) pts[cnt + threadIdx.x] = make_float2(CUDART_INF_F, CUDART_INF_F);
        __syncthreads();
        if (live) {
            const float4* p2 = reinterpret_cast<const float4*>(pts);
            const int quads = (cnt + 3) >> 2;
            // Queries and points are usually numbered along the same curve: the point at the query's relative place is
            // near it, and starting there (a warp at a time) leaves few later points to be inserted.
            int at = (int)((long long)(qi & ~31) * n / nq) - t0;
            at = min(max((at >> 2) - 2, 0), quads - 1);
            for (int z = 0; z < quads; ++z) {
                const float2 d0 = dist2(q.x, q.y, p2[2 * at]), d1 = dist2(q.x, q.y, p2[2 * at + 1]);
                if (fminf(fminf(d0.x, d0.y), fminf(d1.x, d1.y)) <= best[K - 1]) {
                    const float d[4] = {d0.x, d0.y, d1.x, d1.y};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        // (points at an infinite distance, as padding has them, are nobody's neighbours)
                        if (d[i] <= best[K - 1] && d[i] < CUDART_INF_F && 4 * at + i < cnt) insert(d[i], t0 + 4 * at + i);
                }
                at = at + 1 < quads ? at + 1 : 0;
            }
        }
    }
    if (live) {
        const long long o = ((long long)b * nq + qi) * K;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            idx_out[o + i] = who[i];
            if (dist_out) dist_out[o + i] = sqrtf(best[i]);
        }
    }
}

template <int K>
int knn2d_t(const float* query, const float* db, int b, int nq, int n, int64_t* idx_out, float* dist_out,
            cudaStream_t s) {
    const dim3 grid((nq + kKnnThreads - 1) / kKnnThreads, b);
    ScopedKernelTimer timer("knn2d", s);
    knn2d_kernel<K><<<grid, kKnnThreads, 0, s>>>(reinterpret_cast<const float2*>(query),
                                                 reinterpret_cast<const float2*>(db), nq, n, idx_out, dist_out);
    note_launch();
    return check_launch();
}

}  // namespace

int launch_knn2d(const float* query, const float* db, int b, int nq, int n, int k, int64_t* idx_out, float* dist_out,
                 cudaStream_t s) {
    switch (k) {
        case 1: return knn2d_t<1>(query, db, b, nq, n, idx_out, dist_out, s);
        case 2: return knn2d_t<2>(query, db, b, nq, n, idx_out, dist_out, s);
        case 3: return knn2d_t<3>(query, db, b, nq, n, idx_out, dist_out, s);
        case 4: return knn2d_t<4>(query, db, b, nq, n, idx_out, dist_out, s);
        case 5: return knn2d_t<5>(query, db, b, nq, n, idx_out, dist_out, s);
        case 6: return knn2d_t<6>(query, db, b, nq, n, idx_out, dist_out, s);
        case 7: return knn2d_t<7>(query, db, b, nq, n, idx_out, dist_out, s);
        case 8: return knn2d_t<8>(query, db, b, nq, n, idx_out, dist_out, s);
        default: return CLUSTEN_ERR_UNSUPPORTED;
    }
}

}  // namespace clusten
