// Fused local attention (forward): the chain that surrounds CLUSTENQK and CLUSTENAV in the model,
//
//   attn = query x gathered keys  (+ position bias)  (+ mask)  (| blank-token logit)  -> softmax
//   out  = attn x gathered values (+ blank probability x blank value)
//
// (models/aff_transformer.py:117-155 of the reference: QK :120, bias :129-134, mask :136-137, blank token
// :140-141, softmax :142, AV :154, blank value :147,155), in one kernel.  The [b, h, n, m] attention tensor
// never reaches HBM and the neighbour indices are read once.  The separate operators stay the contract of the package;
// this entry point is an opt-in for inference.
//
// A warp takes a tile of 16 rows and some or all heads, finds the tile's distinct groups of 8 neighbours (group_core.cuh)
// and runs through them two at a time with an online softmax.  Everything stays in the lanes' own layout:
//   scores   S[row][slot]: lane (g, t) holds rows g, g + 8 and slots 2t, 2t + 1 of every group
//   bias     the tile's biases, by head, in shared memory as [set of 8 rows][place][row][8 slots]; place 0, which is what
//            the record gives for a group that a row does not name, is minus infinity
//   softmax  maxima and sums over the 4 lanes of a row
//   output   out^T[channel][row] = V^T x P^T: the probabilities are the B operand as they stand
// The bias of an edge is looked up once for several heads (their table entries lie side by side).
// Against a version with signed 64-bit look-ups, the blank logit as scalar products and output rows by shuffles: b64 h8 n1843 bf16 238 -> 226 us,
// b256 h2 n3136 338 -> 330.  More instructions less did not help: keys and values by cp.async and ldmatrix 351 us, look-ups behind a branch 354,
// one CTA of 20 warps per SM on neighbouring tiles (L1 hits 39 -> 51 %) 351.
#include "group_core.cuh"

namespace clusten {
namespace {

constexpr int kFWarps = 4;
// Groups per step of the online softmax; the next step's keys and this step's values are in registers meanwhile.  Two groups at
// five CTAs per SM (96 registers) beat four at four (128): b256 h2 n3136 bf16 0.348 ms against 0.422, and 0.387 for two at four.
constexpr int kChunk = 2;

struct FusedParams {
    const void* q;  const void* k;  const void* v;   // [b, h, n, 32] through strides (elements; k and v share theirs)
    long long q_batch, q_head;  int q_row;
    long long x_batch, x_head;  unsigned x_row;      // x_row in bytes
    const int64_t* idx;                              // [b, n, m]
    const void* bias;                                // [b, h, n, m] or nullptr
    const void* table;  const int64_t* pe_idx;  int table_rows;   // [rows, h], [b, n, m] or nullptr
    const int64_t* mask;                             // [b, n, m] (1 = valid) or nullptr
    const void* blank_k;  const void* blank_v;       // [h, 32] or nullptr
    void* out;                                       // [b, h, n, 32]
    int heads, n, m, R, tiles, parts, per_part;
    unsigned total;
    int wide_idx;                                    // m is a multiple of 8; idx, pe_idx, mask start on 16-byte boundaries
    int pad_cl;
    int vec;                                         // the table entries of all BH heads are read as one word
};

template <typename T, int RT> struct BiasTile {
    static constexpr int kPlace = 64;
    static constexpr int kSet = ((RT > 0 ? RT : kGroupMaxR) + 1) * kPlace;
    static constexpr int kHead = 2 * kSet;                                   // elements per head
};

template <typename T> __device__ __forceinline__ T neg_inf() { return Elem<T>::down(-INFINITY); }
// two neighbouring elements
__device__ __forceinline__ float2 pair_of(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 pair_of(const __half* p) { return __half22float2(*reinterpret_cast<const __half2*>(p)); }
__device__ __forceinline__ float2 pair_of(const __nv_bfloat16* p) {
    const unsigned v = *reinterpret_cast<const unsigned*>(p);
    return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
__device__ __forceinline__ void store_pair(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
template <typename T> __device__ __forceinline__ void store_pair(T* p, T a, T b) {
    *reinterpret_cast<unsigned*>(p) = (unsigned)*reinterpret_cast<unsigned short*>(&a) | (unsigned)*reinterpret_cast<unsigned short*>(&b) << 16;
}
// NV heads' entries of a table row as one word
template <typename T, int NV> struct alignas(sizeof(T) * NV) HeadVec { T v[NV]; };

// Two position-table indices, {lo, hi, lo, hi}; -1: none
template <int RT>
__device__ __forceinline__ int4 load_pair_index(const FusedParams& p, long long at, bool live, int j, int m) {
    int4 v = make_int4(-1, -1, -1, -1);
    const int4* src = reinterpret_cast<const int4*>(p.pe_idx + at);
    if (RT > 0 || p.wide_idx) {
        if (live) v = __ldg(src);
    } else {
        if (live && j < m) *reinterpret_cast<int2*>(&v.x) = __ldg(reinterpret_cast<const int2*>(src));
        if (live && j + 1 < m) *reinterpret_cast<int2*>(&v.z) = __ldg(reinterpret_cast<const int2*>(src) + 1);
    }
    return v;
}
// n 8-byte elements from p on -> L1, without waiting
__device__ __forceinline__ void warm_l1(const int64_t* p, int n, int lane) {
    for (int z = 16 * lane; z < n; z += 512) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p + z));
}

// The position biases of heads h .. h + nh - 1 for the tile -> tile_b[head - h]; slots behind m and place 0: -inf.
// FIRST: also place 0, and the mask: bit 2 r + e of mbits[set]: slot 8 r + 2 t + e of the lane's row is masked out
template <typename T, int RT, int BH, int NV, bool FIRST>
__device__ __forceinline__ void stage_bias(const FusedParams& p, T* tile_b, long long edge0, int rows, int m, int R_arg, int h, int nh, int lane,
                                           unsigned (&mbits)[2]) {
    using B = BiasTile<T, RT>;
    const int R = RT > 0 ? RT : R_arg;
    const int g = lane >> 2, t = lane & 3;
    const char* entries = reinterpret_cast<const char*>(static_cast<const T*>(p.table) + h);
    const unsigned row_bytes = (unsigned)(p.heads * (int)sizeof(T));      // of a table row
    if (FIRST)
        for (int z = lane; z < BH * 2 * 32; z += 32)                         // place 0 of every head and set
            store_pair(tile_b + (z >> 6) * B::kHead + ((z >> 5) & 1) * B::kSet + 2 * (z & 31), neg_inf<T>(), neg_inf<T>());
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const bool live = 8 * e + g < rows;
        const long long at = edge0 + (long long)(8 * e + g) * m + 2 * t;
        T* dst = tile_b + e * B::kSet + B::kPlace + g * 8 + 2 * t;
        unsigned mb = 0u;
#pragma unroll 3
        for (int r = 0; r < R; ++r, dst += B::kPlace) {
            const bool in0 = live && (RT > 0 || 8 * r + 2 * t < m), in1 = live && (RT > 0 || 8 * r + 2 * t + 1 < m);
            int4 v = make_int4(-1, -1, -1, -1);
            if (p.table) v = load_pair_index<RT>(p, at + 8 * r, live, 8 * r + 2 * t, m);
            if (FIRST && p.mask) {
                if (in0 && __ldg(p.mask + at + 8 * r) == 0) mb |= 1u << (2 * r);
                if (in1 && __ldg(p.mask + at + 8 * r + 1) == 0) mb |= 2u << (2 * r);
            }
            const bool ok0 = v.y == 0 && (unsigned)v.x < (unsigned)p.table_rows, ok1 = v.w == 0 && (unsigned)v.z < (unsigned)p.table_rows;
            const T none0 = RT > 0 || in0 ? Elem<T>::down(0.f) : neg_inf<T>(), none1 = RT > 0 || in1 ? Elem<T>::down(0.f) : neg_inf<T>();
            for (int j = 0; j < (NV == BH ? BH : nh); j += NV) {             // (whole words: the heads at hand are all BH of them)
                const char* first = entries + j * (int)sizeof(T);
                HeadVec<T, NV> a, b;
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    a.v[i] = none0;
                    b.v[i] = none1;
                }
                if (ok0) a = *reinterpret_cast<const HeadVec<T, NV>*>(first + (unsigned long long)(unsigned)v.x * row_bytes);
                if (ok1) b = *reinterpret_cast<const HeadVec<T, NV>*>(first + (unsigned long long)(unsigned)v.z * row_bytes);
#pragma unroll
                for (int i = 0; i < NV; ++i) store_pair(dst + (j + i) * B::kHead, a.v[i], b.v[i]);
            }
        }
        if (FIRST) mbits[e] = mb;
    }
    __syncwarp();
}

// Scores of a group are added to d = {row g: slots 2t, 2t + 1; row g + 8: the same}
template <typename T> struct QueryFrag;
template <> struct QueryFrag<float> {
    unsigned h[2][8], l[2][8];                   // rows g, g + 8: channels 4t .. 4t+3, 16+4t .. 16+4t+3
};
struct QueryFrag16 { uint4 r[2]; };              // rows g, g + 8: channels 8t .. 8t+7
template <> struct QueryFrag<__half> : QueryFrag16 {};
template <> struct QueryFrag<__nv_bfloat16> : QueryFrag16 {};

template <typename T> struct KeyRow { uint4 v; };
template <> struct KeyRow<float> { float4 v[2]; };

// (holes: the row may be nullptr, an absent slot)
template <typename T> __device__ __forceinline__ void load_key(KeyRow<T>& k, const char* row, bool holes) {
    if (holes) k.v = make_uint4(0u, 0u, 0u, 0u);
    if (!holes || row) k.v = __ldg(reinterpret_cast<const uint4*>(row));
}
__device__ __forceinline__ void load_key(KeyRow<float>& k, const char* row, bool holes) {
    if (holes) k.v[0] = k.v[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!holes || row) {
        k.v[0] = __ldg(reinterpret_cast<const float4*>(row));
        k.v[1] = __ldg(reinterpret_cast<const float4*>(row) + 4);
    }
}
template <typename T> __device__ __forceinline__ void group_scores(float (&d)[4], const QueryFrag<T>& q, const KeyRow<T>& k) {
    const unsigned a0[4] = {q.r[0].x, q.r[1].x, q.r[0].y, q.r[1].y}, a1[4] = {q.r[0].z, q.r[1].z, q.r[0].w, q.r[1].w};
    const unsigned b0[2] = {k.v.x, k.v.y}, b1[2] = {k.v.z, k.v.w};
    mma16(d, a0, b0, static_cast<const T*>(nullptr));
    mma16(d, a1, b1, static_cast<const T*>(nullptr));
}
__device__ __forceinline__ void group_scores(float (&d)[4], const QueryFrag<float>& q, const KeyRow<float>& k) {
    float e[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float4 kv = k.v[s >> 1];
        const float b[2] = {(s & 1) ? kv.z : kv.x, (s & 1) ? kv.w : kv.y};
        unsigned bh[2], bl[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) split_tf32(b[i], bh[i], bl[i]);
        const unsigned ah[4] = {q.h[0][2 * s], q.h[1][2 * s], q.h[0][2 * s + 1], q.h[1][2 * s + 1]};
        const unsigned al[4] = {q.l[0][2 * s], q.l[1][2 * s], q.l[0][2 * s + 1], q.l[1][2 * s + 1]};
        mma_tf32(d, al, bh);
        if (s == 0) mma_tf32_first(e, ah, bl);
        else mma_tf32(e, ah, bl);
        if (s & 1) mma_tf32(e, ah, bh);
        else mma_tf32(d, ah, bh);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] += e[i];
}

// Online softmax of the lane's rows g, g + 8: probabilities are 2^(x - ref), x the logit in powers of two.  ref starts at the
// blank token's logit and only moves when a logit exceeds it by more than 2^kSlack: the maximum itself is not needed, so the
// usual step has no shuffles.  (A reference above all logits is harmless: it is itself one of the terms.)  Without a blank
// token the first logits that a row meets set its reference.
struct RowState {
    float ref[2];
    float2 sum[2];                               // of the even and of the odd slots
    bool set[2];
};
constexpr float kSlack = 14.f;                   // probabilities are rounded to fp16
constexpr float kLog2e = 1.4426950408889634f;
// (a, b) * f + c and s += (a, b), two at a time
__device__ __forceinline__ void fma_pair(float& a, float& b, float f, float c) {
    asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%0, %1};\nmov.b64 y, {%2, %2};\nmov.b64 z, {%3, %3};\nfma.rn.f32x2 x, x, y, z;\nmov.b64 {%0, %1}, x;\n}\n"
        : "+f"(a), "+f"(b) : "f"(f), "f"(c));
}
__device__ __forceinline__ void add_pair(float2& s, float a, float b) {
    asm("{\n.reg .b64 x, y;\nmov.b64 x, {%0, %1};\nmov.b64 y, {%2, %3};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}\n"
        : "+f"(s.x), "+f"(s.y) : "f"(a), "f"(b));
}

// The groups of one piece for one head.  kx, vx: the head's keys at channel 8t (fp32: 4t; RUNS: at row g) and values as load_rows
// takes them;  bt: the head's bias tile at row g, slot 2t;  dense: dense biases of row g at slot 2t, or nullptr;  act: which sets
// of 8 rows the piece belongs to.  Bound by the L1 (keys 8, values 8 + 8 for their transposition, of 27 cycles per group in
// 16 bits) and the issue slots around it; with values read in the operand's own layout, 16 cycles, b256 h2 n3136 bf16 took
// 0.348 ms against 0.335, b64 h2 n3136 fp32 0.181 against 0.168.
template <typename PICK, typename T, int SET>
__device__ __forceinline__ void attend(const QueryFrag<T>& q, const char* kx, const char* vx, unsigned x_row, const T* bt, const T* dense,
                                       int m, const unsigned (&mbits)[2], bool extra, const GroupSmem& sm, const unsigned short* tok, int U,
                                       bool act0, bool act1, int pad_cl, int n, int lane, RowState& st, float (&acc)[2][2][4]) {
    const int g = lane >> 2, t = lane & 3;
    // the keys of the next groups travel while this step's softmax runs, and so do its values
    KeyRow<T> k[kChunk];
    auto load_keys = [&](int c0) {
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
            load_key(k[i], slot_ptr<PICK>(kx, x_row, sm, tok, c0 + i, g, pad_cl, n), PICK::kHoles);
        }
    };
    load_keys(0);
#pragma unroll 1
    for (int c0 = 0; c0 < U; c0 += kChunk) {
        float x[kChunk][4];
        unsigned rm[2];
        rm[0] = act0 ? *reinterpret_cast<const unsigned short*>(&sm.rec.map[g][c0]) : 0u;
        rm[1] = act1 ? *reinterpret_cast<const unsigned short*>(&sm.rec.map[g + 8][c0]) : 0u;
        // ---- bias + scores
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 bv = pair_of(bt + e * SET + 64 * byte_of(rm[e], i));
                x[i][2 * e] = bv.x;
                x[i][2 * e + 1] = bv.y;
            }
            group_scores(x[i], q, k[i]);
        }
        if (c0 + kChunk < U) load_keys(c0 + kChunk);
        RowRegs<T> w;
        load_rows<PICK>(w, vx, x_row, sm, tok, c0, lane, pad_cl, n);
        if (extra) {                                         // uniform: dense biases, masked slots
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int i = 0; i < kChunk; ++i) {
                    const int place = (int)byte_of(rm[e], i);
                    if (place == 0) continue;
                    float dx = 0.f, dy = 0.f;
                    if (dense) {
                        const T* pb = dense + (long long)(8 * e) * m + 8 * (place - 1);
                        if (8 * (place - 1) + 2 * t < m) dx = Elem<T>::up(pb[0]);
                        if (8 * (place - 1) + 2 * t + 1 < m) dy = Elem<T>::up(pb[1]);
                    }
                    const unsigned mb = mbits[e] >> (2 * (place - 1));
                    if (mb & 1u) dx -= 100.f;
                    if (mb & 2u) dy -= 100.f;
                    x[i][2 * e] += dx;
                    x[i][2 * e + 1] += dy;
                }
        }
        // ---- exponents relative to the rows' references; far above them: move those, and scale what is there down
        float top = st.set[0] && st.set[1] ? -INFINITY : INFINITY;
#pragma unroll
        for (int i = 0; i < kChunk; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                fma_pair(x[i][2 * e], x[i][2 * e + 1], kLog2e, -st.ref[e]);
                top = fmaxf(top, fmaxf(x[i][2 * e], x[i][2 * e + 1]));
            }
        if (__any_sync(kFull, top > kSlack)) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < kChunk; ++i) mx = fmaxf(mx, fmaxf(x[i][2 * e], x[i][2 * e + 1]));
                mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, 2));
                const bool met = mx > -INFINITY;
                const float up = st.set[e] ? fmaxf(mx, 0.f) : (met ? mx : 0.f);
                const float scale = st.set[e] ? exp2f(-up) : 1.f;           // (nothing is there before the reference is set)
                st.set[e] = st.set[e] || met;
                st.ref[e] += up;
                st.sum[e].x *= scale;
                st.sum[e].y *= scale;
#pragma unroll
                for (int i = 0; i < kChunk; ++i) {
                    x[i][2 * e] -= up;
                    x[i][2 * e + 1] -= up;
                }
                const float f0 = __shfl_sync(kFull, scale, 8 * t), f1 = __shfl_sync(kFull, scale, 8 * t + 4);      // rows 2t, 2t + 1
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    acc[e][mt][0] *= f0;  acc[e][mt][1] *= f1;  acc[e][mt][2] *= f0;  acc[e][mt][3] *= f1;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kChunk; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                x[i][2 * e] = exp2f(x[i][2 * e]);
                x[i][2 * e + 1] = exp2f(x[i][2 * e + 1]);
                add_pair(st.sum[e], x[i][2 * e], x[i][2 * e + 1]);
            }
        // ---- output
        rows_product<T, 2>(acc, w, lane, [&](int e, int i) {
            if constexpr (std::is_same<T, float>::value) return make_float2(x[i][2 * e], x[i][2 * e + 1]);
            else return pack2(x[i][2 * e], x[i][2 * e + 1], static_cast<const T*>(nullptr));
        });
    }
}

// The tile's query rows g, g + 8 as operands, and their products with the blank key (nullptr: none), which stands in slot 0 of a group
template <typename T>
__device__ __forceinline__ void load_query(QueryFrag<T>& q, const T* y, int y_row, int rows, const T* blank_k, int g, int t, float (&blank)[2]) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        q.r[e] = make_uint4(0u, 0u, 0u, 0u);
        if (g + 8 * e < rows) q.r[e] = __ldg(reinterpret_cast<const uint4*>(y + (long long)(g + 8 * e) * y_row + 8 * t));
        blank[e] = 0.f;
    }
    if (blank_k) {
        KeyRow<T> k;
        k.v = make_uint4(0u, 0u, 0u, 0u);
        if (g == 0) k.v = __ldg(reinterpret_cast<const uint4*>(blank_k + 8 * t));
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        group_scores(d, q, k);
        blank[0] = __shfl_sync(kFull, d[0], 4 * g);
        blank[1] = __shfl_sync(kFull, d[2], 4 * g);
    }
}
__device__ __forceinline__ void load_query(QueryFrag<float>& q, const float* y, int y_row, int rows, const float* blank_k, int g, int t, float (&blank)[2]) {
    float4 k0 = make_float4(0.f, 0.f, 0.f, 0.f), k1 = k0;
    if (blank_k) {
        k0 = __ldg(reinterpret_cast<const float4*>(blank_k + 4 * t));
        k1 = __ldg(reinterpret_cast<const float4*>(blank_k + 16 + 4 * t));
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
        if (g + 8 * e < rows) {
            const float4* p = reinterpret_cast<const float4*>(y + (long long)(g + 8 * e) * y_row + 4 * t);
            v0 = __ldg(p);
            v1 = __ldg(p + 4);
        }
        const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) split_tf32(v[i], q.h[e][i], q.l[e][i]);
        blank[e] = v0.x * k0.x + v0.y * k0.y + v0.z * k0.z + v0.w * k0.w + v1.x * k1.x + v1.y * k1.y + v1.z * k1.z + v1.w * k1.w;
    }
}

// RT: groups per row known at compile time (m = 48) or 0;  BH: heads whose biases are in shared memory at a time;  TAIL: the last
// cluster is padded
template <typename T, int RT, int BH, bool TAIL>
__global__ void __launch_bounds__(32 * kFWarps, sizeof(T) == 2 ? 5 : 4)
fused_attention_kernel(const __grid_constant__ FusedParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using B = BiasTile<T, RT>;
    constexpr bool kF32 = std::is_same<T, float>::value;
    constexpr int kWarpBytes = (int)sizeof(GroupSmem) + BH * B::kHead * (int)sizeof(T);
    static_assert(BH * B::kHead * (int)sizeof(T) >= kTagSpan, "the tags of build_record fit in the bias tiles");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GroupSmem& sm = *reinterpret_cast<GroupSmem*>(smem_raw + warp * kWarpBytes);
    T* tile_b = reinterpret_cast<T*>(smem_raw + warp * kWarpBytes + sizeof(GroupSmem));
    const unsigned task = blockIdx.x * kFWarps + warp;
    if (task >= p.total) return;
    const unsigned bt = task / (unsigned)p.parts;
    const int part = (int)(task - bt * (unsigned)p.parts);
    const int b = (int)(bt / (unsigned)p.tiles);
    const int i0 = (int)(bt - (unsigned)b * (unsigned)p.tiles) * kTR;
    const int n = p.n, m = RT > 0 ? 8 * RT : p.m;
    const int rows = min(kTR, n - i0);
    const int g = lane >> 2, t = lane & 3;
    const int h0 = part * p.per_part, h1 = min(p.heads, h0 + p.per_part);
    const long long edge0 = ((long long)b * n + i0) * m;
    if (p.table) warm_l1(p.pe_idx + edge0, rows * m, lane);      // (in flight while the record is made)
    if (p.mask) warm_l1(p.mask + edge0, rows * m, lane);
    build_record<RT, TAIL>(p.idx + edge0, rows, m, p.R, n, p.wide_idx != 0, sm.rec, reinterpret_cast<unsigned char*>(tile_b), lane);
    unpack_record<false>(sm, rows, lane);
    const unsigned head = sm.rec.head;
    const unsigned kind = head & 0xffu;
    const int U0 = (head >> 8) & 0xffu;
    unsigned mbits[2] = {0u, 0u};
    const T* Q = static_cast<const T*>(p.q) + (long long)b * p.q_batch + (long long)i0 * p.q_row;
    auto stage = [&](int h, auto first) {
        constexpr bool FIRST = decltype(first)::value;
        const int nh = min(BH, h1 - h);
        if (p.vec) stage_bias<T, RT, BH, BH, FIRST>(p, tile_b, edge0, rows, m, p.R, h, nh, lane, mbits);
        else stage_bias<T, RT, BH, 1, FIRST>(p, tile_b, edge0, rows, m, p.R, h, nh, lane, mbits);
    };
    stage(h0, std::true_type{});
    for (int h = h0; h < h1; ++h) {
        if (h > h0 && (h - h0) % BH == 0) {
            __syncwarp();
            stage(h, std::false_type{});
        }
        const long long bh = (long long)b * p.heads + h;
        const T* bt_h = tile_b + ((h - h0) % BH) * B::kHead + g * 8 + 2 * t;
        const T* dense = p.bias ? static_cast<const T*>(p.bias) + (bh * n + i0 + g) * m + 2 * t : nullptr;
        const T* kx = static_cast<const T*>(p.k) + (long long)b * p.x_batch + (long long)h * p.x_head + (kF32 ? 4 : 8) * t;
        const T* vx = static_cast<const T*>(p.v) + (long long)b * p.x_batch + (long long)h * p.x_head + rows_channel<T>(lane);
        const char* kc = reinterpret_cast<const char*>(kx);
        const char* vc = reinterpret_cast<const char*>(vx);
        QueryFrag<T> q;
        float blank[2];
        load_query(q, Q + (long long)h * p.q_head, p.q_row, rows, p.blank_k ? static_cast<const T*>(p.blank_k) + h * kC : nullptr, g, t, blank);
        RowState st;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (kF32) {                                      // (fp32: the lanes' shares)
                blank[e] += __shfl_xor_sync(kFull, blank[e], 1);
                blank[e] += __shfl_xor_sync(kFull, blank[e], 2);
            }
            blank[e] *= kLog2e;
            st.set[e] = p.blank_k && blank[e] > -INFINITY;   // (no reference: minus infinity, NaN)
            st.ref[e] = st.set[e] ? blank[e] : 0.f;
            st.sum[e] = make_float2(0.f, 0.f);
        }
        float acc[2][2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = acc[1][0][i] = acc[1][1][i] = 0.f;
        const bool extra = dense != nullptr || __any_sync(kFull, (mbits[0] | mbits[1]) != 0u);
        if (kind == kRecRuns) {
            attend<Pick<true, false, TAIL>, T, B::kSet>(q, kc + g * (unsigned long long)p.x_row, vc + rows_first<T>(lane) * (unsigned long long)p.x_row, p.x_row, bt_h,
                                                        dense, m, mbits, extra, sm, sm.tok, U0, true, true, p.pad_cl, n, lane, st, acc);
        } else {
            // one list per 8 rows, or a few rows at a time
            for (int first = 0; first < rows;) {
                int U = U0, take = 8;
                if (kind == kRecOther) take = load_piece<RT>(p.idx + edge0, first, rows, m, n, p.wide_idx != 0, sm, lane, &U);
                const unsigned short* tok = sm.tok + (kind == kRecOther ? 0 : (first >> 3) * kGroupMaxM);
                attend<Pick<false, true>, T, B::kSet>(q, kc, vc, p.x_row, bt_h, dense, m, mbits, extra, sm, tok, U, first < 8, first >= 8, -1, n, lane, st, acc);
                first += take;
            }
        }
        // ---- normalise, add the blank token's share, store rows 2t, 2t + 1 of both sets
        float inv[2], pb[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float sum = st.sum[e].x + st.sum[e].y;
            sum += __shfl_xor_sync(kFull, sum, 1);
            sum += __shfl_xor_sync(kFull, sum, 2);
            const float eb = p.blank_k ? exp2f(blank[e] - st.ref[e]) : 0.f;
            inv[e] = 1.f / (sum + eb);
            pb[e] = eb * inv[e];
        }
        float bv[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        if (p.blank_v) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int i = 0; i < 2; ++i) bv[mt][i] = Elem<T>::up(static_cast<const T*>(p.blank_v)[h * kC + acc_channel<T>(g, mt, i)]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float f = __shfl_sync(kFull, inv[e], 8 * t + 4 * j), fb = __shfl_sync(kFull, pb[e], 8 * t + 4 * j);
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int i = 0; i < 2; ++i) acc[e][mt][2 * i + j] = acc[e][mt][2 * i + j] * f + fb * bv[mt][i];
            }
            T* o = static_cast<T*>(p.out) + (bh * n + i0 + 8 * e) * kC;
            if constexpr (kF32) {
                store_set(acc[e], o, rows - 8 * e, lane);
            } else {
                // a matrix has channels 8w + 2r and 8w + 2r + 1 of the rows, w = 0 .. 3 (frag_slots16): rows of 64 bytes over the head's biases, which are
                // done with (the minus infinities in front of them stay), and a lane takes the four words of its piece
                const T* type = nullptr;
                const unsigned buf = smem_u32(tile_b + ((h - h0) % BH) * B::kHead + B::kPlace);
                __syncwarp();
                stmatrix_x4_trans(buf + row_piece(lane & 7, lane >> 3), pack2(acc[e][0][0], acc[e][0][1], type), pack2(acc[e][0][2], acc[e][0][3], type),
                                  pack2(acc[e][1][0], acc[e][1][1], type), pack2(acc[e][1][2], acc[e][1][3], type));
                __syncwarp();
                if (g < rows - 8 * e)
                    *reinterpret_cast<uint4*>(o + g * kC + 8 * t) = make_uint4(lds32(buf + row_piece(g, 0) + 4 * t), lds32(buf + row_piece(g, 1) + 4 * t),
                                                                              lds32(buf + row_piece(g, 2) + 4 * t), lds32(buf + row_piece(g, 3) + 4 * t));
            }
        }
    }
}

template <typename T>
int fused_t(FusedParams p, int b, cudaStream_t s) {
    p.tiles = group_tiles(p.n);
    p.R = (p.m + 7) / 8;
    const long long tiles = (long long)b * p.tiles;
    if (tiles * p.heads > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    split_heads(tiles, p.heads, &p.parts, &p.per_part);
    p.total = (unsigned)(tiles * p.parts);
    const uintptr_t tables = reinterpret_cast<uintptr_t>(p.idx) | reinterpret_cast<uintptr_t>(p.pe_idx) | reinterpret_cast<uintptr_t>(p.mask);
    p.wide_idx = p.m % 8 == 0 && tables % 16 == 0;
    p.pad_cl = p.n % 8 ? p.n / 8 : -1;
    const bool m48 = p.m == kMmax && p.wide_idx;
    // 16-bit tables: four heads' entries in one 8-byte look-up where a warp has that many heads (b64 h8 n1843: 0.271 ms against
    // 0.296 with two); two otherwise, which leaves more of the L1 to keys and values (b256 h2 n3136: 0.408 ms against 0.497)
    const int bh = sizeof(T) == 2 && p.heads % 4 == 0 && p.per_part % 4 == 0 ? 4 : 2;
    p.vec = p.heads % bh == 0 && p.per_part % bh == 0 && reinterpret_cast<uintptr_t>(p.table) % (bh * sizeof(T)) == 0;
    auto pick = [&](auto heads) {
        constexpr int BH = decltype(heads)::value;
        if (!m48) return fused_attention_kernel<T, 0, BH, true>;
        return p.pad_cl >= 0 ? fused_attention_kernel<T, 6, BH, true> : fused_attention_kernel<T, 6, BH, false>;
    };
    auto kernel = bh == 4 ? pick(std::integral_constant<int, sizeof(T) == 2 ? 4 : 2>{}) : pick(std::integral_constant<int, 2>{});
    const int smem = kFWarps * ((int)sizeof(GroupSmem) + bh * (m48 ? BiasTile<T, 6>::kHead : BiasTile<T, 0>::kHead) * (int)sizeof(T));
    const int fit = resident_ctas(reinterpret_cast<const void*>(kernel), 32 * kFWarps, smem);
    if (fit < 0) return fit;
    ScopedKernelTimer timer("fused_attention", s);
    kernel<<<(p.total + kFWarps - 1) / kFWarps, 32 * kFWarps, smem, s>>>(p);
    note_launch();
    return check_launch();
}

}  // namespace

bool fused_attention_supported(int dtype, int n, int m, int c) {
    if (dtype != CLUSTEN_F32 && dtype != CLUSTEN_F16 && dtype != CLUSTEN_BF16) return false;
    return c == kC && m >= 1 && m <= kMmax && n >= 1 && n <= 65000;
}

int launch_fused_attention(int dtype, const void* q, const void* k, const void* v, const int64_t* idx, const void* bias,
                           const void* table, const int64_t* pe_idx, int table_rows, const int64_t* mask,
                           const void* blank_k, const void* blank_v, void* out, int b, int h, int n, int m,
                           GatherStrides gs, cudaStream_t s) {
    if (gs.x_row == 0) {
        gs.x_batch = (long long)h * n * kC;  gs.x_head = (long long)n * kC;  gs.x_row = kC;
    }
    if (gs.y_row == 0) {
        gs.y_batch = (long long)h * n * kC;  gs.y_head = (long long)n * kC;  gs.y_row = kC;
    }
    FusedParams p{};
    p.q = q;  p.k = k;  p.v = v;  p.idx = idx;  p.bias = bias;  p.table = table;  p.pe_idx = pe_idx;
    p.table_rows = table_rows;  p.mask = mask;  p.blank_k = blank_k;  p.blank_v = blank_v;  p.out = out;
    p.heads = h;  p.n = n;  p.m = m;
    p.q_batch = gs.y_batch;  p.q_head = gs.y_head;  p.q_row = (int)gs.y_row;
    p.x_batch = gs.x_batch;  p.x_head = gs.x_head;  p.x_row = (unsigned)(gs.x_row * dtype_size(dtype));
    switch (dtype) {
        case CLUSTEN_F32: return fused_t<float>(p, b, s);
        case CLUSTEN_F16: return fused_t<__half>(p, b, s);
        case CLUSTEN_BF16: return fused_t<__nv_bfloat16>(p, b, s);
        default: return CLUSTEN_ERR_DTYPE;
    }
}

}  // namespace clusten
