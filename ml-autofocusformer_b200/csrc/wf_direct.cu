// CLUSTENWF forward (and, further down, d_weights) as a plain walk over the neighbours.
//
//   feat_new[b, i, k, :] = sum_j weights[b, i, j, k] * feat[b, nbhd_idx[b, i, j], :]
//
// Half a warp takes one merge row and every lane 4 channels of a 64-channel group: the half fetches the next 16
// neighbours' indices and ic weights one per lane (contiguous, all in flight together) and hands them round by
// shuffles; per neighbour it reads the feature vector (16 bytes per lane in fp32, 256 contiguous bytes per
// row), four in flight at a time, and adds with fp32 FMAs in neighbour order -- the order of the reference's
// loop (clusten/src/clustenwf_cuda_kernel.cu:41-47), which gathers every feature row ic times per output
// element.  Rows are taken in the row order, so the two rows of a warp and the rows of neighbouring warps share
// most of their neighbours and find them in L1.  No shared memory and 64 registers: 32 warps per SM, against 12
// for the tiled kernel (wf_tiles_kernel), whose staging, de-duplication and three-pass TF32 products cost more
// instruction slots than these 16 FMAs per neighbour.  16-bit inputs take it where few weights share a feature row; else kernels of their own below.
#include "group_core.cuh"
#include "tiled.cuh"

namespace clusten {
namespace {

constexpr int kDirectWarps = 8;

struct WfDirectParams {
    const void* W;        // weights [b, n_out, m, ic]
    const void* F;        // feat [b, n, c]
    void* out;            // feat_new [b, n_out, ic, c]
    const int64_t* idx;   // [b, n_out, m]
    const int* order;     // [b, n_out] or nullptr
    int batch, n_out, n, m, c;
};

template <typename T, int ICT, bool C64>
__global__ void __launch_bounds__(32 * kDirectWarps, 4)
wf_forward_direct_kernel(const WfDirectParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, hl = lane & 15;
    const int m = p.m, c = C64 ? 64 : p.c, n = p.n, n_out = p.n_out;
    const unsigned pairs = (unsigned)(n_out + 1) >> 1;
    const unsigned total = (unsigned)p.batch * pairs;
    const unsigned nwarps = gridDim.x * kDirectWarps;
    for (unsigned task = blockIdx.x * kDirectWarps + warp; task < total; task += nwarps) {
        const int b = (int)(task / pairs);
        const int pos = (int)(task - (unsigned)b * pairs) * 2 + half;
        const long long brow = (long long)b * n_out;
        int rq = -1;
        if (pos < n_out) {
            rq = p.order ? p.order[brow + pos] : pos;
            if ((unsigned)rq >= (unsigned)n_out) rq = -1;        // an entry that is no row number: treated as absent
        }
        const int64_t* irow = p.idx + (brow + max(rq, 0)) * m;
        const T* wrow = static_cast<const T*>(p.W) + (brow + max(rq, 0)) * m * ICT;
        const T* Fb = static_cast<const T*>(p.F) + (long long)b * n * c + 4 * hl;
        for (int c0 = 0; c0 < c; c0 += 64) {
            float4 acc[ICT];
#pragma unroll
            for (int k = 0; k < ICT; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int j0 = 0; j0 < m; j0 += 16) {
                // the half's next 16 neighbours, one per lane
                long long my_t = -1;
                if (rq >= 0 && j0 + hl < m) my_t = irow[j0 + hl];
                const int mine = (my_t >= 0 && my_t < n) ? (int)my_t : -1;
                const int cnt = min(16, m - j0);
                // ... and their weights, one neighbour per lane: the row's 16 m bytes are contiguous
                float my_w[ICT];
#pragma unroll
                for (int k = 0; k < ICT; ++k) my_w[k] = 0.f;
                if (rq >= 0 && j0 + hl < m) {
                    if constexpr (ICT == 4) {
                        const float4 v = ld4(wrow + (j0 + hl) * 4);
                        my_w[0] = v.x;  my_w[1] = v.y;  my_w[2] = v.z;  my_w[3] = v.w;
                    } else {
#pragma unroll
                        for (int k = 0; k < ICT; ++k) my_w[k] = Elem<T>::up(wrow[(j0 + hl) * ICT + k]);
                    }
                }
                // four feature vectors in flight at a time (L1 / L2), summed in neighbour order.  A full chunk of
                // valid neighbours -- the rule -- runs without a test per neighbour.
                const bool clean = cnt == 16 && __all_sync(kFull, mine >= 0);
                if (clean) {
#pragma unroll
                    for (int jj = 0; jj < 16; jj += 4) {
                        float4 f[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int t = __shfl_sync(kFull, mine, jj + u, 16);
                            f[u] = ld4(Fb + (unsigned)t * (unsigned)c + c0);
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
#pragma unroll
                            for (int k = 0; k < ICT; ++k) {
                                const float w = __shfl_sync(kFull, my_w[k], jj + u, 16);
                                acc[k].x += w * f[u].x;
                                acc[k].y += w * f[u].y;
                                acc[k].z += w * f[u].z;
                                acc[k].w += w * f[u].w;
                            }
                        }
                    }
                    continue;
                }
                for (int jj = 0; jj < cnt; jj += 4) {
                    float4 f[4];
                    bool ok[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int t = __shfl_sync(kFull, mine, jj + u, 16);
                        ok[u] = jj + u < cnt && t >= 0;
                        if (ok[u]) f[u] = ld4(Fb + (unsigned)t * (unsigned)c + c0);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float w[ICT];
#pragma unroll
                        for (int k = 0; k < ICT; ++k) w[k] = __shfl_sync(kFull, my_w[k], jj + u, 16);
                        if (ok[u]) {
#pragma unroll
                            for (int k = 0; k < ICT; ++k) {
                                acc[k].x += w[k] * f[u].x;
                                acc[k].y += w[k] * f[u].y;
                                acc[k].z += w[k] * f[u].z;
                                acc[k].w += w[k] * f[u].w;
                            }
                        }
                    }
                }
            }
            if (rq >= 0) {
#pragma unroll
                for (int k = 0; k < ICT; ++k)
                    st4(static_cast<T*>(p.out) + ((brow + rq) * ICT + k) * c + c0 + 4 * hl, acc[k]);
            }
        }
    }
}

// 16-bit inputs: out^T[channel][k] = F^T[channel][slot] x W[slot][k] on the tensor cores, a merge row per warp.  Feature rows are
// read as whole 128-byte lines -- lane 8q + s channels 8s .. 8s+7 of slot q of 4, 4 L1 cycles per 512 bytes -- and transposed in
// registers: of the 8 x 8 block whose rows are (slot, half of the 64 channels), movmatrix leaves lane (g, t) = (lane / 4, lane % 4)
// one channel of each half of slot t;  two such blocks, slots 0 .. 3 and 4 .. 7, are byte-permuted into the A operand, k being the
// order 0 4 1 5 2 6 3 7 of the slots, in which the lane fetches the weights.  Bound by the L1 and what it misses:
// b64 n9216 n_out 1843 c128 bf16 178 us (L1 pipe 85 % busy), 284 in the walk above, b128 n_out 784 c64 98 us, 110.
constexpr int kFw16Warps = 4;
struct WfFw16Params {
    const void* W;  const void* F;  void* out;
    const int64_t* idx;  const int* order;
    int n_out, n, m, c;
    unsigned total;                              // batch * n_out
};
template <typename T, int ICT>
__global__ void __launch_bounds__(32 * kFw16Warps, 8)
wf_forward16_kernel(const WfFw16Params p) {
    constexpr int kSteps = kMmax / 16;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned task = blockIdx.x * kFw16Warps + (threadIdx.x >> 5);
    if (task >= p.total) return;
    const unsigned b = task / (unsigned)p.n_out;
    int row = (int)(task - b * (unsigned)p.n_out);
    const long long brow = (long long)b * p.n_out;
    if (p.order) row = p.order[brow + row];
    if ((unsigned)row >= (unsigned)p.n_out) return;          // an entry that is no row number: treated as absent
    const int m = p.m, c = p.c;
    const int64_t* irow = p.idx + (brow + row) * m;
    int tok[2];                                              // slots lane and lane + 32
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const long long v = lane + 32 * i < m ? __ldg(irow + lane + 32 * i) : -1;
        tok[i] = v >= 0 && v < p.n ? (int)v : -1;
    }
    const bool whole = m == kMmax && __all_sync(kFull, tok[0] >= 0 && (tok[1] >= 0 || lane >= 16));
    // first channel of the slots 4 i + lane / 8 (32 bits: n * c is below 2^32)
    constexpr unsigned kGone = 0xffffffffu;
    unsigned at[4 * kSteps];
#pragma unroll
    for (int i = 0; i < 4 * kSteps; ++i) {
        const int tk = __shfl_sync(kFull, tok[i >> 3], (4 * i & 31) + (lane >> 3));
        at[i] = tk >= 0 ? (unsigned)tk * (unsigned)c : kGone;
    }
    unsigned w[kSteps][2];                                   // weights g of the slots t, 4 + t (+ 8) of every 16
    const unsigned short* wrow = static_cast<const unsigned short*>(p.W) + (brow + row) * m * ICT + g;
#pragma unroll
    for (int s = 0; s < kSteps; ++s)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 16 * s + 8 * i + t;
            const unsigned lo = g < ICT && j < m ? __ldg(wrow + j * ICT) : 0u, hi = g < ICT && j + 4 < m ? __ldg(wrow + (j + 4) * ICT) : 0u;
            w[s][i] = lo | hi << 16;
        }
    const T* Fb = static_cast<const T*>(p.F) + (long long)b * p.n * c + 8 * (lane & 7);
    T* o = static_cast<T*>(p.out) + (brow + row) * ICT * c;
    auto channels = [&](int c0, auto check) {
        constexpr bool CHECK = decltype(check)::value;
        float acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            uint4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (CHECK) x[i] = make_uint4(0u, 0u, 0u, 0u);
                if (!CHECK || at[4 * s + i] != kGone) x[i] = __ldg(reinterpret_cast<const uint4*>(Fb + at[4 * s + i] + c0));
            }
            unsigned v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[i][0] = transpose8(x[i].x);  v[i][1] = transpose8(x[i].y);  v[i][2] = transpose8(x[i].z);  v[i][3] = transpose8(x[i].w);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const unsigned a[4] = {__byte_perm(v[0][r], v[1][r], 0x5410), __byte_perm(v[0][r], v[1][r], 0x7632),
                                       __byte_perm(v[2][r], v[3][r], 0x5410), __byte_perm(v[2][r], v[3][r], 0x7632)};
                mma16(acc[r], a, w[s], static_cast<const T*>(nullptr));
            }
        }
        // M tile r: channels 8 (g / 2) + 2r + g % 2 (rows g) and 32 more (rows g + 8), weights 2t, 2t + 1
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float d[2][4], y[8];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                d[r >> 1][2 * (r & 1)] = acc[r][2 * h];
                d[r >> 1][2 * (r & 1) + 1] = acc[r][2 * h + 1];
            }
            acc_rows16(d, lane, y);
            const int k = 2 * t + (g & 1);
            if (k < ICT)
                *reinterpret_cast<uint4*>(o + (long long)k * c + c0 + 32 * h + 8 * (g >> 1)) =
                    make_uint4(pack2(y[0], y[1], static_cast<const T*>(nullptr)), pack2(y[2], y[3], static_cast<const T*>(nullptr)),
                               pack2(y[4], y[5], static_cast<const T*>(nullptr)), pack2(y[6], y[7], static_cast<const T*>(nullptr)));
        }
    };
    for (int c0 = 0; c0 < c; c0 += 64) {
        if (whole) channels(c0, std::false_type{});
        else channels(c0, std::true_type{});
    }
}
template <typename T>
int wf_forward16(const char* label, const WfFw16Params& p, int ic, cudaStream_t s) {
    auto kernel = ic == 4 ? wf_forward16_kernel<T, 4> : (ic == 2 ? wf_forward16_kernel<T, 2> : wf_forward16_kernel<T, 1>);
    ScopedKernelTimer timer(label, s);
    kernel<<<(p.total + kFw16Warps - 1) / kFw16Warps, 32 * kFw16Warps, 0, s>>>(p);
    note_launch();
    return check_launch();
}

// d_weights the same way:  d_weights[b, i, j, k] = <feat[b, nbhd_idx[b, i, j], :], d_feat_new[b, i, k, :]>.
// Half a warp per merge row, 4 channels per lane: the row's ic gradient vectors stay in registers, four
// neighbours' feature vectors are in flight at a time, every lane forms its 4-channel share of 16 dot products -- those of
// 16 / ic neighbours -- and a butterfly over the 16 lanes (each step halves the values a lane keeps) leaves lane l with
// the complete product number l -- neighbour l / ic, weight l % ic -- so that the 16 results are one contiguous 64-byte store.
// fp32 inputs.  (ic = 1 used to take the tiled kernel's three-pass TF32 products: b8 n_out 368 m 40 c 512 183 us, 30 now.)
struct WfDwDirectParams {
    const float* F;       // feat [b, n, c]
    const float* G;       // d_feat_new [b, n_out, ic, c]
    float* out;           // d_weights [b, n_out, m, ic]
    const int64_t* idx;   // [b, n_out, m]
    const int* order;     // [b, n_out] or nullptr
    int batch, n_out, n, m, c;
};

template <int ICT, bool C64>
__global__ void __launch_bounds__(32 * kDirectWarps, 4)
wf_dweights_direct_kernel(const WfDwDirectParams p) {
    constexpr int kNb = 16 / ICT;                // neighbours of a block of 16 products
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, hl = lane & 15;
    const int m = p.m, c = C64 ? 64 : p.c, n = p.n, n_out = p.n_out;
    const unsigned pairs = (unsigned)(n_out + 1) >> 1;
    const unsigned total = (unsigned)p.batch * pairs;
    const unsigned nwarps = gridDim.x * kDirectWarps;
    for (unsigned task = blockIdx.x * kDirectWarps + warp; task < total; task += nwarps) {
        const int b = (int)(task / pairs);
        const int pos = (int)(task - (unsigned)b * pairs) * 2 + half;
        const long long brow = (long long)b * n_out;
        int rq = -1;
        if (pos < n_out) {
            rq = p.order ? p.order[brow + pos] : pos;
            if ((unsigned)rq >= (unsigned)n_out) rq = -1;
        }
        const int64_t* irow = p.idx + (brow + max(rq, 0)) * m;
        const float* grow = p.G + (brow + max(rq, 0)) * ICT * c + 4 * hl;
        const float* Fb = p.F + (long long)b * n * c + 4 * hl;
        float* orow = p.out + (brow + max(rq, 0)) * m * ICT;
        float4 g[ICT];
        if (C64) {
#pragma unroll
            for (int k = 0; k < ICT; ++k) g[k] = *reinterpret_cast<const float4*>(grow + k * c);
        }
        for (int j0 = 0; j0 < m; j0 += 16) {
            long long my_t = -1;
            if (rq >= 0 && j0 + hl < m) my_t = irow[j0 + hl];
            const int mine = (my_t >= 0 && my_t < n) ? (int)my_t : -1;
            const int cnt = min(16, m - j0);
            // kNb neighbours: shares of the 16 products, butterfly, one store.  CHECK: some neighbour of the
            // chunk may be absent or out of range
            auto block = [&](int jj, auto check) {
                constexpr bool CHECK = decltype(check)::value;
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.f;
                for (int c0 = 0; c0 < c; c0 += 64) {
                    if (!C64) {
#pragma unroll
                        for (int k = 0; k < ICT; ++k) g[k] = *reinterpret_cast<const float4*>(grow + k * c + c0);
                    }
#pragma unroll
                    for (int u0 = 0; u0 < kNb; u0 += 4) {
                        float4 f[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int t = __shfl_sync(kFull, mine, (jj + u0 + u) & 15, 16);
                            if (CHECK) {
                                f[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (t >= 0) f[u] = *reinterpret_cast<const float4*>(Fb + (unsigned)t * (unsigned)c + c0);
                            } else {
                                f[u] = *reinterpret_cast<const float4*>(Fb + (unsigned)t * (unsigned)c + c0);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int k = 0; k < ICT; ++k)
                                v[(u0 + u) * ICT + k] += f[u].x * g[k].x + f[u].y * g[k].y + f[u].z * g[k].z + f[u].w * g[k].w;
                    }
                }
                // butterfly: after the step with mask s a lane keeps the half of its values that its bit s selects
#pragma unroll
                for (int s = 8, cntv = 16; s > 0; s >>= 1, cntv >>= 1) {
                    const bool upper = (hl & s) != 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (i < cntv / 2) {
                            const float lo = v[i], hi = v[i + cntv / 2];
                            const float send = upper ? lo : hi, keep = upper ? hi : lo;
                            v[i] = keep + __shfl_xor_sync(kFull, send, s, 16);
                        }
                    }
                }
                // lane l holds product l: neighbour jj + l / ic, weight l % ic
                if (CHECK) {
                    if (rq >= 0 && jj + hl / ICT < cnt) orow[(j0 + jj) * ICT + hl] = v[0];
                } else {
                    orow[(j0 + jj) * ICT + hl] = v[0];
                }
            };
            const bool clean = cnt == 16 && __all_sync(kFull, mine >= 0);      // both rows present, all neighbours valid
            if (clean) {
#pragma unroll
                for (int jj = 0; jj < 16; jj += kNb) block(jj, std::false_type{});
            } else {
                for (int jj = 0; jj < cnt; jj += kNb) block(jj, std::true_type{});
            }
        }
    }
}

// 16-bit inputs: S[slot][k] = F[slot][channel] x G^T[channel][k] on the tensor cores.  A warp takes a merge row; lane (g, t) =
// (lane / 4, lane % 4) reads 8 channels of the slots g, g + 8 of every 16 (the A operand as it stands) and of the gradient of weight
// g (the B operand; columns from ic on are zero).  Every feature row is read once and no lane does more than 2 of its 16-byte
// pieces per product, so the walk is bound by the L1 and what it misses: b128 n_out 784 m 48 c 64 bf16 87 us, 127 in the
// tiled kernel (wf_tiles_kernel).
struct WfDw16Params {
    const void* F;  const void* G;  void* out;
    const int64_t* idx;  const int* order;
    int n_out, n, m, c;
    unsigned total;                              // batch * n_out
};
template <typename T, int ICT>
__global__ void __launch_bounds__(32 * kFw16Warps, 8)
wf_dweights16_kernel(const WfDw16Params p) {
    constexpr int kTiles = kMmax / 16;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const unsigned task = blockIdx.x * kFw16Warps + (threadIdx.x >> 5);
    if (task >= p.total) return;
    const unsigned b = task / (unsigned)p.n_out;
    int row = (int)(task - b * (unsigned)p.n_out);
    const long long brow = (long long)b * p.n_out;
    if (p.order) row = p.order[brow + row];
    if ((unsigned)row >= (unsigned)p.n_out) return;          // an entry that is no row number: treated as absent
    const int m = p.m, c = p.c;
    const int64_t* irow = p.idx + (brow + row) * m;
    int tok[2];                                              // slots lane and lane + 32
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const long long v = lane + 32 * i < m ? __ldg(irow + lane + 32 * i) : -1;
        tok[i] = v >= 0 && v < p.n ? (int)v : -1;
    }
    const T* Fb = static_cast<const T*>(p.F) + (long long)b * p.n * c + 8 * t;
    const T* rows[kTiles][2];
#pragma unroll
    for (int i = 0; i < kTiles; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int tk = __shfl_sync(kFull, tok[(16 * i + 8 * e) >> 5], ((16 * i + 8 * e) & 31) + g);
            rows[i][e] = tk >= 0 ? Fb + (long long)tk * c : nullptr;
        }
    const T* grow = static_cast<const T*>(p.G) + ((brow + row) * ICT + min(g, ICT - 1)) * c + 8 * t;
    float acc[kTiles][4];
#pragma unroll
    for (int i = 0; i < kTiles; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int c0 = 0; c0 < c; c0 += 32) {
        uint4 y = make_uint4(0u, 0u, 0u, 0u), x[kTiles][2];
        if (g < ICT) y = __ldg(reinterpret_cast<const uint4*>(grow + c0));
#pragma unroll
        for (int i = 0; i < kTiles; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                x[i][e] = make_uint4(0u, 0u, 0u, 0u);
                if (rows[i][e]) x[i][e] = __ldg(reinterpret_cast<const uint4*>(rows[i][e] + c0));
            }
        const unsigned b0[2] = {y.x, y.y}, b1[2] = {y.z, y.w};
#pragma unroll
        for (int i = 0; i < kTiles; ++i) {
            const unsigned a0[4] = {x[i][0].x, x[i][1].x, x[i][0].y, x[i][1].y}, a1[4] = {x[i][0].z, x[i][1].z, x[i][0].w, x[i][1].w};
            mma16(acc[i], a0, b0, static_cast<const T*>(nullptr));
            mma16(acc[i], a1, b1, static_cast<const T*>(nullptr));
        }
    }
    // lane (g, t): weights 2t, 2t + 1 of the slots g and g + 8
    T* o = static_cast<T*>(p.out) + (brow + row) * m * ICT;
#pragma unroll
    for (int i = 0; i < kTiles; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = 16 * i + 8 * e + g;
            if (j >= m || 2 * t >= ICT) continue;
            const T lo = Elem<T>::down(acc[i][2 * e]), hi = Elem<T>::down(acc[i][2 * e + 1]);
            if constexpr (ICT == 1) o[j] = lo;
            else *reinterpret_cast<unsigned*>(o + j * ICT + 2 * t) = (unsigned)*reinterpret_cast<const unsigned short*>(&lo) | (unsigned)*reinterpret_cast<const unsigned short*>(&hi) << 16;
        }
}

template <typename T>
int wf_dweights16(const char* label, const WfDw16Params& p, int ic, cudaStream_t s) {
    auto kernel = ic == 4 ? wf_dweights16_kernel<T, 4> : (ic == 2 ? wf_dweights16_kernel<T, 2> : wf_dweights16_kernel<T, 1>);
    ScopedKernelTimer timer(label, s);
    kernel<<<(p.total + kFw16Warps - 1) / kFw16Warps, 32 * kFw16Warps, 0, s>>>(p);
    note_launch();
    return check_launch();
}

template <int ICT>
int wf_dweights_direct(const char* label, const WfDwDirectParams& p, cudaStream_t s) {
    auto kernel = p.c == 64 ? wf_dweights_direct_kernel<ICT, true> : wf_dweights_direct_kernel<ICT, false>;
    const int per_sm = resident_ctas(reinterpret_cast<const void*>(kernel), 32 * kDirectWarps, 0);
    if (per_sm < 0) return per_sm;
    const long long tasks = (long long)p.batch * ((p.n_out + 1) / 2);
    long long grid = (long long)sm_count() * per_sm;
    const long long need = (tasks + kDirectWarps - 1) / kDirectWarps;
    if (grid > need) grid = need;
    ScopedKernelTimer timer(label, s);
    kernel<<<(int)grid, 32 * kDirectWarps, 0, s>>>(p);
    note_launch();
    return check_launch();
}

template <typename T, int ICT>
int wf_forward_direct_t(const char* label, const WfDirectParams& p, cudaStream_t s) {
    auto kernel = p.c == 64 ? wf_forward_direct_kernel<T, ICT, true> : wf_forward_direct_kernel<T, ICT, false>;
    const int per_sm = resident_ctas(reinterpret_cast<const void*>(kernel), 32 * kDirectWarps, 0);
    if (per_sm < 0) return per_sm;
    const long long tasks = (long long)p.batch * ((p.n_out + 1) / 2);
    long long grid = (long long)sm_count() * per_sm;
    const long long need = (tasks + kDirectWarps - 1) / kDirectWarps;
    if (grid > need) grid = need;
    ScopedKernelTimer timer(label, s);
    kernel<<<(int)grid, 32 * kDirectWarps, 0, s>>>(p);
    note_launch();
    return check_launch();
}

}  // namespace

bool wf_forward_direct_supported(int dtype, int n_out, int n, int m, int ic, int c) {
    // element offsets inside a batch element are kept in 32 bits
    return (dtype == CLUSTEN_F32 || dtype == CLUSTEN_F16 || dtype == CLUSTEN_BF16) && (ic == 1 || ic == 2 || ic == 4) &&
           c % 64 == 0 &&
           (long long)n * c <= 0xffffffffLL && (long long)n_out * m * ic <= 0x7fffffffLL;
}

template <typename T>
static int wf_forward_direct_ic(const char* label, int ic, const WfDirectParams& p, cudaStream_t s) {
    switch (ic) {
        case 1: return wf_forward_direct_t<T, 1>(label, p, s);
        case 2: return wf_forward_direct_t<T, 2>(label, p, s);
        case 4: return wf_forward_direct_t<T, 4>(label, p, s);
        default: return CLUSTEN_ERR_UNSUPPORTED;
    }
}

int launch_wf_forward_direct(const char* label, int dtype, const void* W, const void* F, const int64_t* idx,
                             const int* order, void* out, int b, int n_out, int n, int m, int ic, int c,
                             cudaStream_t s) {
    // 16-bit: the tensor-core kernel does the work of 48 slots and 8 weights whatever there are, and more of it per row before the first channels; the walk's work
    // grows with m and ic.  us, walk / tensor cores: c 64 (b128 n3136 n_out 784) ic 1 m 48 60 / 95, m 24 40 / 93, ic 2 79 / 94, 54 / 85, ic 4 111 / 103,
    // 75 / 89;  c 256 ic 1 232 / 264, 153 / 245, ic 2 295 / 257, 201 / 218, ic 4 450 / 281, 299 / 239;  c 512 m 48 ic 1 462 / 494, ic 2 596 / 482.
    // The walk needs warps (half a one per row): b128 n_out 50 c 64 ic 1 6.8 / 9.1, b8 n_out 196 5.1 / 4.7, c 512 18.9 / 13.3
    const bool walk = m * ic <= (c == 64 ? 96 : 48) && (long long)b * n_out >= 32LL * sm_count();
    if (dtype != CLUSTEN_F32 && (long long)b * n_out > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    if (dtype != CLUSTEN_F32 && !walk) {
        WfFw16Params p{};
        p.W = W;  p.F = F;  p.out = out;  p.idx = idx;  p.order = order;
        p.n_out = n_out;  p.n = n;  p.m = m;  p.c = c;  p.total = (unsigned)b * n_out;
        return dtype == CLUSTEN_F16 ? wf_forward16<__half>(label, p, ic, s) : wf_forward16<__nv_bfloat16>(label, p, ic, s);
    }
    WfDirectParams p{};
    p.W = W;  p.F = F;  p.out = out;  p.idx = idx;  p.order = order;
    p.batch = b;  p.n_out = n_out;  p.n = n;  p.m = m;  p.c = c;
    if ((long long)b * ((n_out + 1) / 2) > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    switch (dtype) {
        case CLUSTEN_F32: return wf_forward_direct_ic<float>(label, ic, p, s);
        case CLUSTEN_F16: return wf_forward_direct_ic<__half>(label, ic, p, s);
        case CLUSTEN_BF16: return wf_forward_direct_ic<__nv_bfloat16>(label, ic, p, s);
        default: return CLUSTEN_ERR_DTYPE;
    }
}

int launch_wf_dweights_direct(const char* label, int dtype, const void* F, const void* G, const int64_t* idx, const int* order,
                              void* d_weights, int b, int n_out, int n, int m, int ic, int c, cudaStream_t s) {
    if ((long long)b * n_out > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    if (dtype != CLUSTEN_F32) {
        WfDw16Params p{};
        p.F = F;  p.G = G;  p.out = d_weights;  p.idx = idx;  p.order = order;
        p.n_out = n_out;  p.n = n;  p.m = m;  p.c = c;  p.total = (unsigned)b * n_out;
        return dtype == CLUSTEN_F16 ? wf_dweights16<__half>(label, p, ic, s) : wf_dweights16<__nv_bfloat16>(label, p, ic, s);
    }
    WfDwDirectParams p{};
    p.F = static_cast<const float*>(F);  p.G = static_cast<const float*>(G);  p.out = static_cast<float*>(d_weights);
    p.idx = idx;  p.order = order;
    p.batch = b;  p.n_out = n_out;  p.n = n;  p.m = m;  p.c = c;
    switch (ic) {
        case 1: return wf_dweights_direct<1>(label, p, s);
        case 2: return wf_dweights_direct<2>(label, p, s);
        case 4: return wf_dweights_direct<4>(label, p, s);
        default: return CLUSTEN_ERR_UNSUPPORTED;
    }
}

}  // namespace clusten
