// Scatter side of QK / AV (d_key, d_value; head_dim 32) over an inverse index by target tile (group_inverse.cu):
//
//   out[b, h, t, :] = sum over (i, j) with nbhd_idx[b, i, j] == t of  W[b, h, i, j] * X[b, h, i, :]
//
// A warp takes the 8 targets 8T .. 8T+7 of a batch element and some or all heads and forms
// out^T[channel][target] = X^T[channel][row] * W[row][target] on the tensor cores (FP32 inputs as TF32 in three passes).
// 16-bit, whole clusters and lists: scatter_runs16, scatter_lists16.  Else lane (g, t) = (lane / 4, lane % 4) reads 4 channels of the rows whose products it
// feeds, and the weights of those rows for target 8T + g: in an AutoFocusFormer table the 8 targets of a row that names the cluster
// are 8 neighbouring weights, so a request covers 4 rows times 16 or 32 contiguous bytes, and rows that do not name it are not read at
// all.  Operands go from L1 / L2 into registers; no de-duplication, no atomics, a fixed order of summation.
//   16-bit: one m16n8k16 step is 16 entries; fp32: two steps of 8 rows.
// Batch elements with the ordinary index (random tables) take the targets one after the other, 16 (8) entries per step.
//
// The reference adds every (row, slot, channel) term with atomicAdd (clusten/src/clustenqk_cuda_kernel.cu:117-127,
// clustenav_cuda_kernel.cu:113-123).
#include "group_core.cuh"

namespace clusten {
namespace {

constexpr int kSGWarps = 4;

struct ScatterGroupsParams {
    const void* W;  long long w_batch, w_head;  int w_row;      // [b,h,n,m] (element strides)
    const void* X;  long long x_batch, x_head;  int x_row;      // [b,h,n,32]
    const int64_t* idx;                                         // [b,n,m]
    InverseView inv;
    void* out;                                                  // [b,h,n,32], contiguous
    int heads, n, m, parts, per_part;
    unsigned total;                                             // batch * ntiles * parts
    unsigned m_magic, m_shift;                                  // x / m = (umulhi(magic, x) + x) >> shift
};

// Products of the rows r[i] (nullptr: none) with the weights w[i] (nullptr: zero).  16-bit: 4 rows per lane, one step;
// fp32: 2 rows per lane.
__device__ __forceinline__ unsigned ldw16(const void* p) { return p ? (unsigned)__ldg(static_cast<const unsigned short*>(p)) : 0u; }
template <typename T>
__device__ __forceinline__ void step16(float (&acc)[2][4], const T* const (&r)[4], const T* const (&w)[4]) {
    uint2 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = make_uint2(0u, 0u);
        if (r[i]) x[i] = __ldg(reinterpret_cast<const uint2*>(r[i]));
    }
    const unsigned b[2] = {ldw16(w[0]) | ldw16(w[1]) << 16, ldw16(w[2]) | ldw16(w[3]) << 16};
    unsigned a[2][4];
    frag_channels16(a, x[0], x[1], x[2], x[3]);
    mma16(acc[0], a[0], b, static_cast<const T*>(nullptr));
    mma16(acc[1], a[1], b, static_cast<const T*>(nullptr));
}
// (FIRST: d starts at zero)
template <bool FIRST>
__device__ __forceinline__ void step8(float (&d)[2][4], const float* const (&r)[2], const float* const (&w)[2]) {
    float4 x[2];
    float b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r[i]) x[i] = __ldg(reinterpret_cast<const float4*>(r[i]));
        b[i] = w[i] ? __ldg(w[i]) : 0.f;
    }
    const float a[2][4] = {{x[0].x, x[0].y, x[1].x, x[1].y}, {x[0].z, x[0].w, x[1].z, x[1].w}};
    if (FIRST) mma_pair_first(d, a, b);
    else mma_pair<true>(d, a, b);
}
// rows and weights of 16 rows (4 per lane).  ALONE, fp32: the products of a step are added up by themselves and then to the accumulator:
// a tensor core cuts its sums off, and over the hundreds of rows that name a cluster the cut adds up (2-norm error against 64 bits
// of d_key, d_value, straight into the accumulator and so: b8 h8 n196 7.7e-7 -> 4.5e-7, b4 h8 n1843 7.5e-7 -> 4.5e-7, b8 h2 n3136
// 7.4e-7 -> 4.5e-7).  The lists of shared tables are short; there the extra registers cost 8 % of a training pass.
template <typename T, bool ALONE>
__device__ __forceinline__ void step_rows(float (&acc)[2][4], const T* const (&r)[4], const T* const (&w)[4]) {
    if constexpr (std::is_same<T, float>::value) {
        const float* const ra[2] = {r[0], r[1]};
        const float* const wa[2] = {w[0], w[1]};
        const float* const rb[2] = {r[2], r[3]};
        const float* const wb[2] = {w[2], w[3]};
        if constexpr (ALONE) {
            float d[2][4];
            step8<true>(d, ra, wa);
            step8<false>(d, rb, wb);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[0][i] += d[0][i];
                acc[1][i] += d[1][i];
            }
        } else {
            step8<false>(acc, ra, wa);
            step8<false>(acc, rb, wb);
        }
    } else {
        step16<T>(acc, r, w);
    }
}

// ----------------------------------------------------------------------------- whole clusters, 16-bit
// A step is 16 entries of the tile's list.  Its 16 rows of X (64 bytes each) and the 16 x 8 weights travel to shared memory by
// cp.async, kSDepth - 1 steps ahead and across the warp's heads, and come back as operands by ldmatrix.trans.  The entries
// behind the last one (place 0) are filled with zeros without a look at memory.  Against rows and weights that went from L1 straight
// into operand registers: b128 h2 n3136 bf16 121 -> 97 us, b32 h8 n1843 fp16 111 -> 63, b128 h8 n196 bf16 62 -> 34 (in the last two
// one more walk over the padded cluster's list instead of one per padded slot).  Bound by the L1 (83 % busy, b64 h2 n3136): a row of X or of
// weights is a line of its own.
constexpr int kSDepth = 2;                        // (3: the same times with 20 % more shared memory; 4: b128 h2 n3136 bf16 120 us, for want of L1)
template <bool SHIFT> struct RunsStage {
    static constexpr int kW = 16 * 64;                       // 16 rows of X (row_piece)
    static constexpr int kAt = kW + 16 * (SHIFT ? 32 : 16);  // weights; SHIFT (rows start anywhere): the two aligned pieces that cover them,
    static constexpr int kBytes = kAt + (SHIFT ? 32 : 0);    // and at which byte of them the first one is
    static constexpr int kWarp = kSDepth * kBytes;
};

// acc: channels g, g + 8 (and 16, 24 more) of targets 2t, 2t + 1 -> the tile's rows, by way of the stage at buf, whose operands have been read
template <typename T> __device__ __forceinline__ void store_targets(const float (&acc)[2][4], unsigned buf, T* out, int rows, int lane) {
    const int g = lane >> 2, t = lane & 3;
    __syncwarp();
    acc_to_rows<T>(acc, buf, lane);
    __syncwarp();
    if (g < rows) *reinterpret_cast<uint4*>(out + g * kC + 8 * t) = lds128(buf + row_piece(g, t));
}

// sm: the warp's RunsStage::kWarp bytes;  list, own: the tile's entries and its steps;  pad_list, pad: those of the padded cluster, whose
// slots from `first_pad` on name token 0 (tile 0 only; else pad = 0);  w, x: of the first head;  out: the tile's rows there
template <typename T, bool SHIFT, bool TAIL>
__device__ __forceinline__ void scatter_runs16(unsigned char* sm, const unsigned* list, int own, const unsigned* pad_list, int pad, int first_pad,
                                               int heads, const T* w, long long w_head, int w_row, const T* x, long long x_head, int x_row, T* out,
                                               long long out_head, int rows, int lane) {
    using S = RunsStage<SHIFT>;
    const int g = lane >> 2, t = lane & 3;
    const unsigned base = smem_u32(sm);
    const int per_head = pad + own;
    // ---- copies: rows lane / 4 and 8 + lane / 4, piece lane % 4
    const unsigned x_dst = base + row_piece(g, t);
    const char* xi = reinterpret_cast<const char*>(x) + 16 * t;
    const unsigned x_bytes = 2u * (unsigned)x_row;
    const T* wi = w - 8;
    int left = per_head * heads, step = 0;
    unsigned next = left > 0 ? __ldg((pad > 0 ? pad_list : list) + (lane & 15)) : 0u;
    unsigned stage = 0u;
    auto issue = [&]() {
        if (left > 0) {
            const unsigned e = next;
            const char* xh = xi;
            const T* wh = wi;
            --left;
            if (++step == per_head) {
                step = 0;
                xi += 2 * x_head;
                wi += w_head;
            }
            if (left > 0) next = __ldg((TAIL && step < pad ? pad_list + 16 * step : list + 16 * (step - pad)) + (lane & 15));
            const unsigned e0 = __shfl_sync(kFull, e, g), e1 = __shfl_sync(kFull, e, 8 + g);
            cp_async16_or_zero(x_dst + stage, xh + (unsigned long long)(e0 >> 8) * x_bytes, (e0 & 255u) != 0u);
            cp_async16_or_zero(x_dst + stage + 512, xh + (unsigned long long)(e1 >> 8) * x_bytes, (e1 & 255u) != 0u);
            if (SHIFT) {
                const unsigned ew = __shfl_sync(kFull, e, lane >> 1);
                const uintptr_t at = reinterpret_cast<uintptr_t>(wh + (unsigned long long)(ew >> 8) * (unsigned)w_row + 8 * (ew & 255u));
                const unsigned off = (unsigned)at & 15u;
                const bool there = (ew & 255u) != 0u && ((lane & 1) == 0 || off != 0u);
                cp_async16_or_zero(base + stage + S::kW + 16 * lane, reinterpret_cast<const void*>((at & ~uintptr_t(15)) + 16 * (lane & 1)), there);
                if ((lane & 1) == 0)
                    asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(base + stage + S::kAt + lane), "h"((unsigned short)(16 * lane + off)) : "memory");
            } else if (lane < 16) {
                cp_async16_or_zero(base + stage + S::kW + 16 * lane, wh + (unsigned long long)(e >> 8) * (unsigned)w_row + 8 * (e & 255u), (e & 255u) != 0u);
            }
            stage = stage == (kSDepth - 1) * S::kBytes ? 0u : stage + S::kBytes;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int d = 0; d < kSDepth - 1; ++d) issue();
    // ---- products
    const int r = (lane & 7) + 8 * (lane >> 4), c = (lane >> 3) & 1;
    const unsigned a_at = base + row_piece(r, c), a_at2 = base + row_piece(r, c + 2);
    unsigned now = 0u;
    for (int h = 0; h < heads; ++h) {
        float acc[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][i] = acc[1][i] = 0.f;
        for (int s = 0; s < per_head; ++s) {
            cp_async_wait<kSDepth - 2>();
            __syncwarp();
            issue();
            unsigned a[2][4], bw[2];
            ldmatrix_x4_trans(a[0], a_at + now);
            ldmatrix_x4_trans(a[1], a_at2 + now);
            if (SHIFT) {
                const unsigned o0 = lds32(base + now + S::kAt + 4 * t), o1 = lds32(base + now + S::kAt + 16 + 4 * t);
                const unsigned wb = base + now + S::kW + 2 * g;
                bw[0] = lds16(wb + (o0 & 0xffffu)) | lds16(wb + (o0 >> 16)) << 16;
                bw[1] = lds16(wb + (o1 & 0xffffu)) | lds16(wb + (o1 >> 16)) << 16;
            } else {
                ldmatrix_x2_trans(bw, base + now + S::kW + 16 * (lane & 15));
            }
            mma16(acc[0], a[0], bw, static_cast<const T*>(nullptr));
            mma16(acc[1], a[1], bw, static_cast<const T*>(nullptr));
            now = now == (kSDepth - 1) * S::kBytes ? 0u : now + S::kBytes;
            if (TAIL && s == pad - 1) {
                // the padded slots are all token 0: their columns -> column 0
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    float* d = &acc[i >> 2][i & 3];
                    float sum = (2 * t >= first_pad ? d[0] : 0.f) + (2 * t + 1 >= first_pad ? d[1] : 0.f);
                    sum += __shfl_xor_sync(kFull, sum, 1);
                    sum += __shfl_xor_sync(kFull, sum, 2);
                    d[0] = t == 0 ? sum : 0.f;
                    d[1] = 0.f;
                }
            }
        }
        store_targets<T>(acc, base + (now == 0u ? (kSDepth - 1) * S::kBytes : now - S::kBytes), out, rows, lane);
        out += out_head;
    }
    cp_async_wait<0>();
}

// Lists, 16-bit: a step is two entries, 8 + 8 rows; the rows travel as above, the weights -- one slot for each target, wherever it lies in the row --
// one step ahead into the registers of the lanes that feed them.  Training passes over tables shared by a cluster, d_query and d_key / d_attn and
// d_value: b128 h2 n3136 bf16 216, 232 -> 200, 205 us, b64 h8 n784 m24 98, 97 -> 76, 82.  ents: the tile's entries, `count` of them
template <typename T, int STAGE>
__device__ __forceinline__ void scatter_lists16(unsigned char* sm, const uint4* ents, int count, int heads, const T* w, long long w_head, int w_row, const T* x,
                                                long long x_head, int x_row, T* out, long long out_head, int n, int rows, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const unsigned base = smem_u32(sm), x_dst = base + row_piece(g, t), x_bytes = 2u * (unsigned)x_row;
    const char* xi = reinterpret_cast<const char*>(x) + 16 * t;
    const T* wi = w;
    const int per_head = (count + 1) >> 1;
    int left = per_head * heads, step = 0;
    const uint4 none = make_uint4((unsigned)n, 0xffffffffu, 0xffffffffu, 0u);
    uint4 e[2] = {none, none};
    auto load = [&](int s) {
        e[0] = __ldg(ents + 2 * s);
        e[1] = 2 * s + 1 < count ? __ldg(ents + 2 * s + 1) : none;
    };
    if (left > 0) load(0);
    unsigned stage = 0u, coming[2] = {0u, 0u};
    auto issue = [&]() {
        if (left > 0) {
            const char* xh = xi;
            const T* wh = wi;
            const uint4 now[2] = {e[0], e[1]};
            --left;
            if (++step == per_head) {
                step = 0;
                xi += 2 * x_head;
                wi += w_head;
            }
            if (left > 0) load(step);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const unsigned row = now[z].x + g;
                cp_async16_or_zero(x_dst + stage + 512 * z, xh + (unsigned long long)(row < (unsigned)n ? row : 0u) * x_bytes, row < (unsigned)n);
                const unsigned j = ((g & 4 ? now[z].z : now[z].y) >> (8 * (g & 3))) & 0xffu;
                unsigned v[2] = {0u, 0u};
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const unsigned r = now[z].x + 2 * t + i;
                    if (j != 0xffu && r < (unsigned)n) v[i] = __ldg(reinterpret_cast<const unsigned short*>(wh + (unsigned long long)r * (unsigned)w_row + j));
                }
                coming[z] = v[0] | v[1] << 16;
            }
            stage = stage == (kSDepth - 1) * STAGE ? 0u : stage + STAGE;
        }
        cp_async_commit();
    };
    static_assert(kSDepth == 2, "the weights are one step ahead");
    issue();
    const int r = (lane & 7) + 8 * (lane >> 4), c = (lane >> 3) & 1;
    const unsigned a_at = base + row_piece(r, c), a_at2 = base + row_piece(r, c + 2);
    unsigned now = 0u;
    for (int h = 0; h < heads; ++h) {
        float acc[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][i] = acc[1][i] = 0.f;
        for (int s = 0; s < per_head; ++s) {
            const unsigned bw[2] = {coming[0], coming[1]};
            cp_async_wait<0>();
            __syncwarp();
            issue();
            unsigned a[2][4];
            ldmatrix_x4_trans(a[0], a_at + now);
            ldmatrix_x4_trans(a[1], a_at2 + now);
            mma16(acc[0], a[0], bw, static_cast<const T*>(nullptr));
            mma16(acc[1], a[1], bw, static_cast<const T*>(nullptr));
            now = STAGE - now;
        }
        store_targets<T>(acc, base + STAGE - now, out, rows, lane);
        out += out_head;
    }
    cp_async_wait<0>();
}

template <typename T, bool M48, bool TAIL, bool SHIFT>
__global__ void __launch_bounds__(32 * kSGWarps, 8)
scatter_groups_kernel(const __grid_constant__ ScatterGroupsParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned task = blockIdx.x * kSGWarps + warp;
    if (task >= p.total) return;
    const unsigned bt = task / (unsigned)p.parts;
    const int part = (int)(task - bt * (unsigned)p.parts);
    const int b = (int)(bt / (unsigned)p.inv.ntiles);
    const int tile = (int)(bt - (unsigned)b * (unsigned)p.inv.ntiles);
    const int n = p.n, m = M48 ? 48 : p.m;
    const int g = lane >> 2, t = lane & 3;
    const int h0 = part * p.per_part, h1 = min(p.heads, h0 + p.per_part);
    const int mode = __ldg(p.inv.tileflag + (long long)b * (1 + p.inv.ntiles));
    const int* rowptr = p.inv.rowptr + (long long)b * (n + 1);
    const int* seglen = p.inv.seglen + (long long)b * n;
    const uint4* ents = group_entries(p.inv.entries, b, n, m);
    const T* Wb = static_cast<const T*>(p.W) + (long long)b * p.w_batch;
    const T* Xb = static_cast<const T*>(p.X) + (long long)b * p.x_batch + 4 * g;
    int start = 0, count = 0;
    if (mode != kBuildGeneral) {
        start = __ldg(rowptr + tile);
        count = __ldg(seglen + tile);
    }
    if constexpr (sizeof(T) == 2) {
        unsigned char* sm = smem_raw + warp * RunsStage<SHIFT>::kWarp;
        const T* W0 = Wb + (long long)h0 * p.w_head;
        const T* X0 = static_cast<const T*>(p.X) + (long long)b * p.x_batch + (long long)h0 * p.x_head;
        T* out0 = static_cast<T*>(p.out) + (((long long)b * p.heads + h0) * n + tile * 8) * kC;
        if (mode == kBuildGroupRuns) {
            int pad_start = 0, pad_count = 0;
            if (TAIL && tile == 0) {
                pad_start = __ldg(rowptr + (n >> 3));
                pad_count = __ldg(seglen + (n >> 3));
            }
            const unsigned* list = reinterpret_cast<const unsigned*>(ents);
            scatter_runs16<T, SHIFT, TAIL>(sm, list + start, count >> 4, list + pad_start, pad_count >> 4, n & 7, h1 - h0, W0, p.w_head, p.w_row, X0, p.x_head, p.x_row, out0,
                                           (long long)n * kC, n - tile * 8, lane);
            return;
        }
        if (mode == kBuildGroupLists) {
            scatter_lists16<T, RunsStage<SHIFT>::kBytes>(sm, ents + start, count, h1 - h0, W0, p.w_head, p.w_row, X0, p.x_head, p.x_row, out0, (long long)n * kC, n, n - tile * 8, lane);
            return;
        }
    }
    for (int h = h0; h < h1; ++h) {
        const T* W = Wb + (long long)h * p.w_head;
        const T* X = Xb + (long long)h * p.x_head;
        float acc[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][i] = acc[1][i] = 0.f;
        if (sizeof(T) == 4 && mode == kBuildGroupRuns) {
            // 16 rows a step, 4 per lane, the next step's entries on their way
            const T* Wg = W + g - 8;
            auto walk = [&](const uint4* list, int steps, const T* w0, bool live) {
                uint4 e = steps > 0 ? __ldg(list + t) : make_uint4(0u, 0u, 0u, 0u);
                for (int k = 0; k < steps; ++k) {
                    const unsigned ee[4] = {e.x, e.y, e.z, e.w};
                    if (k + 1 < steps) e = __ldg(list + 4 * (k + 1) + t);
                    const T* r[4];
                    const T* w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const unsigned row = ee[i] >> 8, place = ee[i] & 255u;
                        r[i] = place ? X + (long long)row * p.x_row : nullptr;
                        w[i] = place && live ? w0 + (long long)row * p.w_row + 8 * place : nullptr;
                    }
                    step_rows<T, true>(acc, r, w);
                }
            };
            walk(ents + (start >> 2), count >> 4, Wg, true);
            if (TAIL && tile == 0) {
                // the slots that pad the last cluster name token 0
                const int last = n >> 3, s1 = __ldg(rowptr + last), c1 = __ldg(seglen + last);
                for (int q = n & 7; q < 8; ++q) walk(ents + (s1 >> 2), c1 >> 4, Wg + q, g == 0);
            }
        } else if (sizeof(T) == 4 && mode == kBuildGroupLists) {
            // two entries of 8 rows per step: rows t and t + 4 of each
            uint4 e[2];
            auto load = [&](int k) {
#pragma unroll
                for (int z = 0; z < 2; ++z) e[z] = k + z < count ? __ldg(ents + start + k + z) : make_uint4((unsigned)n, 0xffffffffu, 0xffffffffu, 0u);
            };
            load(0);
            for (int k = 0; k < count; k += 2) {
                const T* r[4];
                const T* w[4];
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const unsigned j = ((g & 4 ? e[z].z : e[z].y) >> (8 * (g & 3))) & 0xffu;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int row = (int)e[z].x + t + 4 * i;
                        const bool live = row < n;
                        r[2 * z + i] = live ? X + (long long)row * p.x_row : nullptr;
                        w[2 * z + i] = live && j != 0xffu ? W + (long long)row * p.w_row + j : nullptr;
                    }
                }
                if (k + 2 < count) load(k + 2);
                step_rows<T, false>(acc, r, w);
            }
        } else {
            // the ordinary index: target by target, 16 entries per step
            const int* entries = p.inv.entries + (long long)b * n * m;
            for (int q = 0; q < 8 && tile * 8 + q < n; ++q) {
                const int tgt = tile * 8 + q;
                const int s0 = __ldg(rowptr + tgt), len = __ldg(seglen + tgt);
                for (int k = 0; k < len; k += 16) {
                    const T* r[4];
                    const T* w[4];
                    bool repeats = false;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int at = k + 4 * i + t;
                        r[i] = w[i] = nullptr;
                        if (at < len) {
                            const unsigned e = (unsigned)__ldg(entries + s0 + at);
                            if (e & kDupFlag) {
                                repeats = true;                // the row names the target more than once: below
                            } else {
                                const unsigned row = M48 ? e / 48u : (__umulhi(p.m_magic, e) + e) >> p.m_shift;
                                r[i] = X + (long long)row * p.x_row;
                                if (g == q) w[i] = W + (long long)row * p.w_row + (e - row * (unsigned)m);
                            }
                        }
                    }
                    step_rows<T, false>(acc, r, w);
                    if (__any_sync(kFull, repeats)) {
                        // the row's weights for the target are added up in fp32, in slot order
                        for (int z = k; z < min(k + 16, len); ++z) {
                            const unsigned e = (unsigned)__ldg(entries + s0 + z);
                            if (!(e & kDupFlag)) continue;     // uniform
                            const unsigned row = (e & ~kDupFlag) / (unsigned)m;
                            const int64_t* irow = p.idx + ((long long)b * n + row) * m;
                            float sum = 0.f;
                            for (int j = 0; j < m; ++j)
                                if (__ldg(irow + j) == tgt) sum += Elem<T>::up(W[(long long)row * p.w_row + j]);
                            if (t == q >> 1) {
                                const float4 x = ld4(X + (long long)row * p.x_row);
                                const int c = q & 1;
                                acc[0][c] += sum * x.x;
                                acc[0][c + 2] += sum * x.y;
                                acc[1][c] += sum * x.z;
                                acc[1][c + 2] += sum * x.w;
                            }
                        }
                    }
                }
            }
        }
        T* o = static_cast<T*>(p.out) + (((long long)b * p.heads + h) * n + tile * 8 + 2 * t) * kC + 4 * g;
        if (tile * 8 + 2 * t < n) st4(o, acc_channels(acc, 0));
        if (tile * 8 + 2 * t + 1 < n) st4(o + kC, acc_channels(acc, 1));
    }
}

template <typename T>
int scatter_groups_t(const char* label, ScatterGroupsParams p, cudaStream_t s) {
    constexpr int kPer = 16 / (int)sizeof(T);
    const bool shift = sizeof(T) == 2 && (reinterpret_cast<uintptr_t>(p.W) % 16 != 0 || p.w_row % kPer != 0 || p.w_batch % kPer != 0 || p.w_head % kPer != 0);
    auto pick = [&](auto m48, auto tail) {
        constexpr bool M48 = decltype(m48)::value, TAIL = decltype(tail)::value;
        return shift ? scatter_groups_kernel<T, M48, TAIL, sizeof(T) == 2> : scatter_groups_kernel<T, M48, TAIL, false>;
    };
    auto kernel = p.n & 7 ? (p.m == 48 ? pick(std::true_type{}, std::true_type{}) : pick(std::false_type{}, std::true_type{}))
                          : (p.m == 48 ? pick(std::true_type{}, std::false_type{}) : pick(std::false_type{}, std::false_type{}));
    const int smem = sizeof(T) == 2 ? kSGWarps * (shift ? RunsStage<true>::kWarp : RunsStage<false>::kWarp) : 0;
    const int fit = resident_ctas(reinterpret_cast<const void*>(kernel), 32 * kSGWarps, smem);
    if (fit < 0) return fit;
    ScopedKernelTimer timer(label, s);
    kernel<<<(p.total + kSGWarps - 1) / kSGWarps, 32 * kSGWarps, smem, s>>>(p);
    note_launch();
    return check_launch();
}

}  // namespace

// W, X through their strides (gs.y: W, gs.x: X); inv: built by launch_group_inverse
int launch_scatter_groups(const char* label, int dtype, const void* W, const void* X, const int64_t* idx, const InverseView& inv,
                          void* out, int b, int h, int n, int m, const GatherStrides& gs, cudaStream_t s) {
    ScatterGroupsParams p{};
    p.W = W;  p.w_batch = gs.y_batch;  p.w_head = gs.y_head;  p.w_row = (int)gs.y_row;
    p.X = X;  p.x_batch = gs.x_batch;  p.x_head = gs.x_head;  p.x_row = (int)gs.x_row;
    p.idx = idx;  p.inv = inv;  p.out = out;
    p.heads = h;  p.n = n;  p.m = m;
    const long long tiles = (long long)b * inv.ntiles;
    if (tiles * h > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    // 16-bit warps have little to read before the first head: more of them (b32 h8 n1843 fp16 63 us, 70 with 24 per SM; b128 h8 n196 bf16 33, 37).  The ordinary
    // index, whose warps go target by target, gains most: d_query and d_key of random tables b32 h8 n1843 bf16 1707 us, 2456 with 24, b64 h8 n784 2061, 3128
    split_heads(tiles, h, &p.parts, &p.per_part, dtype == CLUSTEN_F32 ? 24 : 64);
    p.total = (unsigned)(tiles * p.parts);
    while ((1ull << p.m_shift) < (unsigned)m) ++p.m_shift;
    p.m_magic = (unsigned)(((1ull << 32) * ((1ull << p.m_shift) - (unsigned)m)) / (unsigned)m + 1);
    switch (dtype) {
        case CLUSTEN_F32: return scatter_groups_t<float>(label, p, s);
        case CLUSTEN_F16: return scatter_groups_t<__half>(label, p, s);
        case CLUSTEN_BF16: return scatter_groups_t<__nv_bfloat16>(label, p, s);
        default: return CLUSTEN_ERR_DTYPE;
    }
}

}  // namespace clusten
