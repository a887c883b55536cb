// Gather side of QK / AV (head_dim 32, m <= 64, in fp32 m <= 48):
//
//   sum   out[i,:] = sum_j W[i,j] * X[idx[i,j],:]          AV forward, d_query
//   dot   out[i,j] = <X[idx[i,j],:], Y[i,:]>               QK forward, d_attn
//
// A warp takes a tile of 16 consecutive rows of one batch element and some or all of its heads, takes the tile's
// distinct groups of 8 neighbours from its record (group_core.cuh) and multiplies them on the tensor cores with
// operands that go from L1 / L2 straight into registers:
//
//   sum   out^T[channel][row] = X^T[channel][slot] * W^T[slot][row].  A lane reads 4 channels of the 4 (fp32: 2)
//         slots whose products it feeds and uses them for both sets of 8 rows; the tile's weights are copied to shared
//         memory as they lie (one contiguous block) and read back one pair per row and group; a row that does not name
//         the group reads the zeros in front of its weights.  The accumulators are 4 channels of two rows.
//   dot   16-bit: S[row][slot] = Y[row][channel] * X^T[channel][slot], 8 channels of one slot per lane.  fp32: S^T, the
//         slots of two groups times 8 rows, so that the three TF32 passes split every neighbour row once.  The scores
//         are laid out by row in shared memory (those of rows that do not name the group in front of them, where nobody
//         looks) and leave as contiguous 16-byte pieces.
//
// 16-bit tiles of whole clusters share their rows with the three next ones (blocks of 64 rows, below).
// FP32 inputs are multiplied as TF32 in three passes (tile_core.cuh), FP16 / BF16 inputs with m16n8k16.
// The reference gives each output element a thread that re-gathers its neighbour rows from L2
// (clusten/src/clustenav_cuda_kernel.cu:18-50, clustenqk_cuda_kernel.cu:18-49).
#include "group_core.cuh"

namespace clusten {
namespace {

constexpr int kGWarps = 4;                       // warps per CTA, independent of each other

struct GatherGroupsParams {
    const void* A;  long long a_batch, a_head;  int a_row;       // sum: W [b,h,n,m], dot: Y [b,h,n,32] (element strides)
    const void* X;  long long x_batch, x_head;  unsigned x_row;  // [b,h,n,32]; x_row in bytes
    const int64_t* idx;                                          // [b,n,m]
    const TileRecord* plan;                                      // [b][tiles] or nullptr: the warps make the records themselves
    void* out;                                                   // sum: [b,h,n,32], dot: [b,h,n,m], contiguous
    int heads, n, m, R, tiles;
    int parts, per_part;                                         // head ranges a tile is split into
    unsigned total;                                              // batch * tiles * parts
    int wide_idx;                                                // m is a multiple of 8, idx starts on a 16-byte boundary
    int pad_cl;                                                  // the cluster that is padded with token 0, or -1
};

// Weight (sum) or score (dot) tile of a warp: [set of 8 rows][place][row of the set][8 slots].  Place 0 belongs to no group;
// group r of a row (place r + 1 in the record) lies at place r + 1.  Whatever places the rows of a set ask for, lane (g, t)
// reads and writes the banks 4g + t (fp32: the pair 8g + 2t of a half warp), so there are no bank conflicts.
// A shifted tile (SHIFT: rows that do not start on 16-byte boundaries) holds the aligned 16-byte pieces that cover a row,
// one place more.
template <typename T, int RT, bool SHIFT> struct RowTile {
    static constexpr int kPlace = 64;                                      // elements of a place: 8 rows x 8 slots
    static constexpr int kSet = ((RT > 0 ? RT : kGroupMaxR) + (SHIFT ? 2 : 1)) * kPlace;
    static constexpr int kBytes = 2 * kSet * (int)sizeof(T);
};
static_assert(RowTile<float, 6, false>::kBytes >= kTagSpan && RowTile<__half, 6, false>::kBytes >= kTagSpan, "the tags of build_record fit in the tile");

// ----------------------------------------------------------------------------- sum
// The tile's weight rows -> shared memory, asynchronously, 16 bytes at a time; neighbouring lanes take neighbouring rows, so
// that they write different banks.
template <typename T, int RT, bool SHIFT>
__device__ __forceinline__ void stage_rows(const T* __restrict__ w, int a_row, int rows, int m, int R, T* buf, int lane) {
    using Tile = RowTile<T, RT, SHIFT>;
    constexpr int kPer = 16 / (int)sizeof(T);                              // elements of a piece
    constexpr int kPieces = 8 / kPer;                                      // pieces of a group: 1 or 2
    const int piece = lane % kPieces, g = (lane / kPieces) & 7;
    constexpr int kStep = 32 / (8 * kPieces);                              // (set, group) pairs per pass: 4 or 2
    const int groups = RT > 0 ? RT + (SHIFT ? 1 : 0) : R + (SHIFT ? 1 : 0);
    constexpr int kMost = 2 * ((RT > 0 ? RT : kGroupMaxR) + (SHIFT ? 1 : 0));
#pragma unroll
    for (int k = 0; k < (kMost + kStep - 1) / kStep; ++k) {
        const int sg = lane / (8 * kPieces) + kStep * k;
        const int e = sg >= groups ? 1 : 0, r = sg - e * groups, row = 8 * e + g;
        if (r < groups && row < rows) {
            T* dst = buf + e * Tile::kSet + (r + 1) * Tile::kPlace + g * 8 + piece * kPer;
            const T* src = w + (long long)row * a_row;
            if (SHIFT) {
                const uintptr_t first = reinterpret_cast<uintptr_t>(src);
                const uintptr_t at = (first & ~uintptr_t(15)) + (8 * r + piece * kPer) * sizeof(T);
                if (at < first + m * sizeof(T)) cp_async16_cg(dst, reinterpret_cast<const void*>(at));       // holds an element of the row
            } else {
                cp_async16_cg(dst, src + 8 * r + piece * kPer);
            }
        }
    }
    cp_async_commit();
}

// Where lane t finds the slots 2t and 2t + 1 of a group of a row that starts at w (element offsets from the row's first
// piece), and by how many bits a 16-bit pair is shifted
struct PairAt {
    int first, second;
    unsigned bits;
};
template <typename T> __device__ __forceinline__ PairAt pair_at(const T* w, int t) {
    PairAt p;
    const int s = (int)((reinterpret_cast<uintptr_t>(w) & 15) / sizeof(T));      // elements between the piece's and the row's start
    if (sizeof(T) == 2) {
        const int q = t + (s >> 1);                                              // 4-byte words
        p.first = (q >> 2) * 64 + (q & 3) * 2;
        p.second = ((q + 1) >> 2) * 64 + ((q + 1) & 3) * 2;
        p.bits = (s & 1) * 16;
    } else {
        const int q = 2 * t + s;
        p.first = (q >> 3) * 64 + (q & 7);
        p.second = ((q + 1) >> 3) * 64 + ((q + 1) & 7);
        p.bits = 0u;
    }
    return p;
}

// One head, NS sets of 8 rows.  x: the head's rows at channel 4g (RUNS: row 2t; fp32 lists without holes: as load_rows takes them);  w: the first set's weights at row g (SHIFT: slot 0 of the
// pieces, at: where the pairs are; else slot 2t);  map: the record's row g of the first set
template <typename PICK, typename T, bool SHIFT, int NS, int SET>
__device__ __forceinline__ void sum_head(const T* __restrict__ x, unsigned x_row, const T* w, const PairAt (&at)[NS], const unsigned char* map,
                                         const GroupSmem& sm, const unsigned short* tok, int U, int pad_cl, int n, int t,
                                         float (&acc)[NS][2][4]) {
    bool landed = false;
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 4) {
        unsigned rm[NS];
#pragma unroll
        for (int e = 0; e < NS; ++e) rm[e] = *reinterpret_cast<const unsigned*>(map + 8 * e * kMaxU + u0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && u0 + 2 >= U) break;
            Four_t<T> v[4];
            unsigned tk[2];
            // fp32, one set of rows (lists): whole rows, as the L1 likes them, moved to their lanes (b128 h2 n3136 146 -> 138 us)
            constexpr bool kWhole = std::is_same<T, float>::value && NS == 1 && !PICK::kRuns && !PICK::kHoles;
            RowRegs<T> whole;
            if constexpr (kWhole) load_rows<PICK>(whole, reinterpret_cast<const char*>(x), x_row, sm, tok, u0 + 2 * h, threadIdx.x & 31, pad_cl, n);
            else load_four<PICK, T>(v, reinterpret_cast<const char*>(x), x_row, sm, tok, u0 + 2 * h, t, pad_cl, n, tk);
            if (!landed) {                                   // the weights travelled together with the first rows
                cp_async_wait<0>();
                __syncwarp();
                landed = true;
            }
            if constexpr (kWhole) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = to_slots(whole.v[i], threadIdx.x & 31);
            }
            if constexpr (std::is_same<T, float>::value) {
                auto weights = [&](int e, int i, float (&bb)[2]) {
                    const unsigned place = byte_of(rm[e], 2 * h + i);
                    const float* p = w + e * SET + 64 * place;
                    float2 q;
                    if (SHIFT) {
                        q.x = place ? p[at[e].first] : 0.f;
                        q.y = place ? p[at[e].second] : 0.f;
                    } else {
                        q = *reinterpret_cast<const float2*>(p);
                    }
                    bb[0] = PICK::kHoles && (tk[i] & 0xffffu) == kSkip ? 0.f : q.x;
                    bb[1] = PICK::kHoles && (tk[i] >> 16) == kSkip ? 0.f : q.y;
                };
                const float a0[2][4] = {{v[0].x, v[0].y, v[1].x, v[1].y}, {v[0].z, v[0].w, v[1].z, v[1].w}};
                const float a1[2][4] = {{v[2].x, v[2].y, v[3].x, v[3].y}, {v[2].z, v[2].w, v[3].z, v[3].w}};
#pragma unroll
                for (int e = 0; e < NS; ++e) {
                    float b[2];
                    weights(e, 0, b);
                    mma_pair<true>(acc[e], a0, b);
                    weights(e, 1, b);
                    mma_pair<true>(acc[e], a1, b);
                }
            } else {
                auto weights = [&](int e, int i) -> unsigned {
                    const unsigned place = byte_of(rm[e], 2 * h + i);
                    const T* p = w + e * SET + 64 * place;
                    unsigned q;
                    if (SHIFT) {
                        q = __funnelshift_r(*reinterpret_cast<const unsigned*>(p + at[e].first), *reinterpret_cast<const unsigned*>(p + at[e].second), at[e].bits);
                        if (place == 0u) q = 0u;
                    } else {
                        q = *reinterpret_cast<const unsigned*>(p);
                    }
                    if (PICK::kHoles && (tk[i] & 0xffffu) == kSkip) q &= 0xffff0000u;
                    if (PICK::kHoles && (tk[i] >> 16) == kSkip) q &= 0xffffu;
                    return q;
                };
                unsigned a[2][4];
                frag_channels16(a, v[0], v[1], v[2], v[3]);
#pragma unroll
                for (int e = 0; e < NS; ++e) {
                    const unsigned b[2] = {weights(e, 0), weights(e, 1)};
                    mma16(acc[e][0], a[0], b, static_cast<const T*>(nullptr));
                    mma16(acc[e][1], a[1], b, static_cast<const T*>(nullptr));
                }
            }
        }
    }
}

// fp32 rows of their own (tables without locality), m <= 48: a lane takes 4 channels of every fourth neighbour, so that a load brings four
// neighbour rows, and the next row's indices and weights travel meanwhile.  Plain FMAs: 2-norm error against 64 bits 1e-7, where
// the TF32 passes have 6.6e-7.  src, w, out: the tile's first row;  x: the head's rows
__device__ __noinline__ void sum_walk(const int64_t* __restrict__ src, const float* __restrict__ w, int a_row, const char* __restrict__ x, unsigned x_row,
                                      float* __restrict__ out, int rows, int m, int n, int lane) {
    const int q = lane >> 3;
    x += 16 * (lane & 7);
    int tok[2];                                              // slots lane, lane + 32 (-1: absent, its weight 0)
    float my_w[2];
    auto load = [&](int row) {
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const int j = lane + 32 * z;
            const long long v = row < rows && j < m ? __ldg(src + (long long)row * m + j) : -1;
            const bool there = (unsigned long long)v < (unsigned long long)n;
            tok[z] = there ? (int)v : -1;
            my_w[z] = there ? __ldg(w + (long long)row * a_row + j) : 0.f;
        }
    };
    load(0);
    for (int row = 0; row < rows; ++row) {
        const int t0 = tok[0], t1 = tok[1];
        const float w0 = my_w[0], w1 = my_w[1];
        load(row + 1);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j0 = 0; j0 < kMmax; j0 += 16) {
            if (j0 >= m) break;
            float4 xv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = __shfl_sync(kFull, j0 < 32 ? t0 : t1, ((j0 + 4 * i) & 31) + q);
                xv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t >= 0) xv[i] = __ldg(reinterpret_cast<const float4*>(x + (unsigned long long)(unsigned)t * x_row));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float wv = __shfl_sync(kFull, j0 < 32 ? w0 : w1, ((j0 + 4 * i) & 31) + q);
                acc.x += wv * xv[i].x;
                acc.y += wv * xv[i].y;
                acc.z += wv * xv[i].z;
                acc.w += wv * xv[i].w;
            }
        }
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            acc.x += __shfl_xor_sync(kFull, acc.x, o);
            acc.y += __shfl_xor_sync(kFull, acc.y, o);
            acc.z += __shfl_xor_sync(kFull, acc.z, o);
            acc.w += __shfl_xor_sync(kFull, acc.w, o);
        }
        if (q == 0) st4(out + (long long)row * kC + 4 * lane, acc);
    }
}

// ----------------------------------------------------------------------------- dot
// Scores of rows whose length is no multiple of 8 lie in the tile as they will in the output, row after row and starting as
// far behind a 16-byte boundary as the output does, so that they leave as 16-byte pieces.  (Taken from the places of the usual
// layout, element by element with a division each, they cost more than the products: b256 h16 n49 m49 bf16 43.5 us, 35.5 us so.)
struct LinearRows {
    int m, left;                                 // slots of a row, and how many of them from the lane's first one on
};
// 16-bit, one head, NS sets of 8 rows: q: Y rows g (and g + 8), channels 8t .. 8t+7;  x: the head's rows at channel 8t (RUNS:
// row g);  o: the first set's scores at row g, slot 2t;  map: the record's row g of the first set;  lin: see LinearRows
template <typename PICK, typename T, int NS, int SET, bool LIN>
__device__ __forceinline__ void dot_head16(const uint4 (&q)[NS], const T* __restrict__ x, unsigned x_row, T* o, const unsigned char* map,
                                           const GroupSmem& sm, const unsigned short* tok, int U, int pad_cl, int n, int g, LinearRows lin) {
    unsigned a0[4] = {q[0].x, 0u, q[0].y, 0u}, a1[4] = {q[0].z, 0u, q[0].w, 0u};
    if (NS == 2) {
        a0[1] = q[NS - 1].x;  a0[3] = q[NS - 1].y;  a1[1] = q[NS - 1].z;  a1[3] = q[NS - 1].w;
    }
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 4) {
        uint4 k[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= 2 && u0 + 2 >= U) break;
            const char* row = slot_ptr<PICK>(reinterpret_cast<const char*>(x), x_row, sm, tok, u0 + i, g, pad_cl, n);
            if (PICK::kHoles) k[i] = make_uint4(0u, 0u, 0u, 0u);
            if (!PICK::kHoles || row) k[i] = __ldg(reinterpret_cast<const uint4*>(row));
        }
        unsigned rm[NS];
#pragma unroll
        for (int e = 0; e < NS; ++e) rm[e] = *reinterpret_cast<const unsigned*>(map + 8 * e * kMaxU + u0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= 2 && u0 + 2 >= U) break;
            float d[4];
            const unsigned b0[2] = {k[i].x, k[i].y}, b1[2] = {k[i].z, k[i].w};
            mma16_first(d, a0, b0, static_cast<const T*>(nullptr));
            mma16(d, a1, b1, static_cast<const T*>(nullptr));
#pragma unroll
            for (int e = 0; e < NS; ++e) {
                const int place = (int)byte_of(rm[e], i);
                if constexpr (LIN) {
                    const int j = 8 * (place - 1);
                    T* row = o + 8 * e * lin.m + j;
                    if (place != 0 && j < lin.left) row[0] = Elem<T>::down(d[2 * e]);
                    if (place != 0 && j + 1 < lin.left) row[1] = Elem<T>::down(d[2 * e + 1]);
                } else {
                    *reinterpret_cast<unsigned*>(o + e * SET + 64 * place) = pack2(d[2 * e], d[2 * e + 1], static_cast<const T*>(nullptr));
                }
            }
        }
    }
}

// fp32: a row's channels 4t .. 4t+3 and 16+4t .. 16+4t+3 as TF32 high and low parts
struct SplitRow {
    unsigned h[8], l[8];
};
__device__ __forceinline__ void load_split(SplitRow& q, const float* y, bool live) {
    float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
    if (live) {
        q0 = __ldg(reinterpret_cast<const float4*>(y));
        q1 = __ldg(reinterpret_cast<const float4*>(y) + 4);
    }
    const float v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) split_tf32(v[i], q.h[i], q.l[i]);
}
// The slots of two groups are the 16 rows of A.  x: the head's rows at channel 4t (RUNS: row g);  o: the first set's scores at row 2t, slot g;
// map: the record's row 2t of the first set
template <typename PICK, int NS, int SET, bool LIN>
__device__ __forceinline__ void dot_head32(const SplitRow (&q)[NS], const float* __restrict__ x, unsigned x_row, float* o,
                                           const unsigned char* map, const GroupSmem& sm, const unsigned short* tok, int U, int pad_cl, int n,
                                           int g, LinearRows lin) {
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 2) {
        float4 k[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const char* row = slot_ptr<PICK>(reinterpret_cast<const char*>(x), x_row, sm, tok, u0 + i, g, pad_cl, n);
            if (PICK::kHoles) k[i][0] = k[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!PICK::kHoles || row) {
                const float4* p = reinterpret_cast<const float4*>(row);
                k[i][0] = __ldg(p);
                k[i][1] = __ldg(p + 4);
            }
        }
        float d[NS][2][4];                                               // [set of rows][chain]
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const float4 ka = k[0][s >> 1], kb = k[1][s >> 1];
            const float av[4] = {(s & 1) ? ka.z : ka.x, (s & 1) ? kb.z : kb.x, (s & 1) ? ka.w : ka.y, (s & 1) ? kb.w : kb.y};
            unsigned ah[4], al[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split_tf32(av[i], ah[i], al[i]);
#pragma unroll
            for (int e = 0; e < NS; ++e) {
                const unsigned bh[2] = {q[e].h[2 * s], q[e].h[2 * s + 1]}, bl[2] = {q[e].l[2 * s], q[e].l[2 * s + 1]};
                if (s == 0) {
                    mma_tf32_first(d[e][0], al, bh);
                    mma_tf32_first(d[e][1], ah, bl);
                } else {
                    mma_tf32(d[e][0], al, bh);
                    mma_tf32(d[e][1], ah, bl);
                }
                mma_tf32(d[e][s & 1], ah, bh);
            }
        }
        // d: slot g of group u0 (0, 1) and u0 + 1 (2, 3) for the rows 2t (0, 2) and 2t + 1 (1, 3)
#pragma unroll
        for (int e = 0; e < NS; ++e)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const unsigned mm = *reinterpret_cast<const unsigned short*>(map + (8 * e + j) * kMaxU + u0);
                const float s0 = d[e][0][j] + d[e][1][j], s1 = d[e][0][j + 2] + d[e][1][j + 2];
                if constexpr (LIN) {
                    const int j0 = 8 * ((int)(mm & 0xffu) - 1), j1 = 8 * ((int)(mm >> 8) - 1);
                    float* row = o + (8 * e + j) * lin.m;
                    if (j0 >= 0 && j0 < lin.left) row[j0] = s0;
                    if (j1 >= 0 && j1 < lin.left) row[j1] = s1;
                } else {
                    float* row = o + e * SET + 8 * j;
                    row[64 * (mm & 0xffu)] = s0;
                    row[64 * (mm >> 8)] = s1;
                }
            }
    }
}

// The scores of all rows -> out (row stride m, rows one after the other).  LIN: LinearRows
template <typename T, int RT, bool LIN>
__device__ __forceinline__ void store_rows(const T* tile, T* __restrict__ out, int rows, int m, int R, int lane) {
    using Tile = RowTile<T, RT, false>;
    constexpr int kPer = 16 / (int)sizeof(T);
    if constexpr (!LIN) {
        constexpr int kPieces = 8 / kPer;
        const int groups = RT > 0 ? RT : R;
        const int piece = lane % kPieces, g = (lane / kPieces) & 7;
        constexpr int kStep = 32 / (8 * kPieces);
#pragma unroll
        for (int k = 0; k < (2 * (RT > 0 ? RT : kGroupMaxR) + kStep - 1) / kStep; ++k) {
            const int sg = lane / (8 * kPieces) + kStep * k;
            const int e = sg >= groups ? 1 : 0, r = sg - e * groups, row = 8 * e + g;
            if (r < groups && row < rows)
                *reinterpret_cast<uint4*>(out + row * m + 8 * r + piece * kPer) =
                    *reinterpret_cast<const uint4*>(tile + e * Tile::kSet + (r + 1) * Tile::kPlace + g * 8 + piece * kPer);
        }
    } else {
        // tile and out start at the same offset inside a 16-byte piece
        const int first = (int)((reinterpret_cast<uintptr_t>(out) & 15) / sizeof(T)), last = first + rows * m;
        const T* src = tile - first;
        T* dst = out - first;
        for (int z = kPer * lane; z < last; z += kPer * 32) {
            if (z >= first && z + kPer <= last) {
                *reinterpret_cast<uint4*>(dst + z) = *reinterpret_cast<const uint4*>(src + z);
            } else {
                for (int i = max(z, first); i < min(z + kPer, last); ++i) dst[i] = src[i];
            }
        }
    }
}

// ----------------------------------------------------------------------------- the kernel
// MODE 0: sum, 1: dot;  RT: groups per row known at compile time (6: m = 48, every AutoFocusFormer stage) or 0;
// SHIFT: the rows of the weights (sum) or scores (dot, LinearRows) do not start on 16-byte boundaries;  PLAN: the records are there;
// TAIL: the last cluster is padded
// CTAs per SM, measured for b128 h2 n3136.  dot: fp32 over records 7 (0.115 ms a call, 0.130 with 5), 5 where the records are made here
// (b4 h2 n9216 22 us, 24 with 6); 16-bit 4, without spills (91 us, 102 with 6; b128 h8 n196 23.2, 25.2; shared tables 99, 94).  sum: fp32 over records
// 5, 6 where they are made here (shared tables 134 us, 138 with 5; b128 h8 n196 45, 50 with 5), 16-bit 7.
template <typename T, int MODE, bool PLAN> constexpr int gather_ctas() {
    if (MODE == 1) return sizeof(T) == 4 ? (PLAN ? 7 : 5) : 4;
    return sizeof(T) == 4 ? (PLAN ? 5 : 6) : 7;
}
// Blocks (below), us with 6 (5, 7), b128 h2 n3136 bf16: dot 61 (64, 59), sum 62 (66, 62), of the model's views 70 (75, 72); b64 h8 n784 30 (33, 30), 31 (36, 34);
// tables shared by a cluster, tile by tile inside: dot 82 (76, 87), b32 h8 n1843 53 (46, 63), sum 63 (67, 65), 41 (41, 39)
constexpr int kBlockCtas = 6;
template <typename T, int MODE, int RT, bool SHIFT, bool PLAN, bool TAIL>
__global__ void __launch_bounds__(32 * kGWarps, (gather_ctas<T, MODE, PLAN>()))
gather_groups_kernel(const __grid_constant__ GatherGroupsParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Tile = RowTile<T, RT, SHIFT>;
    constexpr bool kF32 = std::is_same<T, float>::value;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* base = smem_raw + warp * (int)(sizeof(GroupSmem) + Tile::kBytes);
    GroupSmem& sm = *reinterpret_cast<GroupSmem*>(base);
    T* tile = reinterpret_cast<T*>(base + sizeof(GroupSmem));
    const unsigned task = blockIdx.x * kGWarps + warp;
    if (task >= p.total) return;
    const unsigned bt = task / (unsigned)p.parts;
    const int part = (int)(task - bt * (unsigned)p.parts);
    const int b = (int)(bt / (unsigned)p.tiles);
    const int i0 = (int)(bt - (unsigned)b * (unsigned)p.tiles) * kTR;
    const int n = p.n, m = RT > 0 ? 8 * RT : p.m;
    const int rows = min(kTR, n - i0);
    const int g = lane >> 2, t = lane & 3;
    const int h0 = part * p.per_part, h1 = min(p.heads, h0 + p.per_part);
    const T* A = static_cast<const T*>(p.A) + (long long)b * p.a_batch + (long long)i0 * p.a_row;
    const T* X = static_cast<const T*>(p.X) + (long long)b * p.x_batch + (MODE == 0 ? 4 * g : (kF32 ? 4 : 8) * t);
    const int64_t* src = p.idx + ((long long)b * n + i0) * m;
    if (PLAN) {
        reinterpret_cast<uint4*>(&sm.rec)[lane] = __ldg(reinterpret_cast<const uint4*>(p.plan + bt) + lane);
    } else {
        build_record<RT, TAIL>(src, rows, m, p.R, n, p.wide_idx != 0, sm.rec, reinterpret_cast<unsigned char*>(tile), lane);
    }
    if (MODE == 0) {
        if (!SHIFT) {                                        // the zeros of place 0
            for (int z = lane; z < 2 * Tile::kPlace * (int)sizeof(T) / 16; z += 32) {
                constexpr int kPer = 16 / (int)sizeof(T);
                const int e = z / (Tile::kPlace / kPer), c = z % (Tile::kPlace / kPer);
                *reinterpret_cast<uint4*>(tile + e * Tile::kSet + c * kPer) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        stage_rows<T, RT, SHIFT>(A + (long long)h0 * p.a_head, p.a_row, rows, m, p.R, tile, lane);
    }
    // (16-bit sums: 0 * Inf would be a NaN; three-pass products of infinities are NaN anyway)
    constexpr bool kFill = MODE == 1 || kF32;
    unpack_record<kFill>(sm, rows, lane);
    const unsigned head = sm.rec.head;
    const unsigned kind = head & 0xffu;
    const bool holes = (head >> 16 & (kFill ? 1u : 3u)) != 0u;
    const int U0 = (head >> 8) & 0xffu;
    auto at_row = [&](const T* x, int row) { return reinterpret_cast<const T*>(reinterpret_cast<const char*>(x) + (unsigned long long)row * p.x_row); };
    for (int h = h0; h < h1; ++h) {
        const long long bh = (long long)b * p.heads + h;
        const T* Ah = A + (long long)h * p.a_head;
        const T* Xh = X + (long long)h * p.x_head;
        if constexpr (MODE == 0) {
            if (h > h0) {                                    // (the first head's weights were requested above)
                __syncwarp();
                stage_rows<T, RT, SHIFT>(Ah, p.a_row, rows, m, p.R, tile, lane);
            }
            if constexpr (kF32) {
                if (kind == kRecOther) {
                    cp_async_wait<0>();                      // (the weights that were requested are not used)
                    sum_walk(src, Ah, p.a_row, reinterpret_cast<const char*>(Xh - 4 * g), p.x_row,
                             static_cast<float*>(p.out) + (bh * n + i0) * kC, rows, m, n, lane);
                    continue;
                }
            }
            const T* w = tile + g * 8 + (SHIFT ? 0 : 2 * t);
            T* o = static_cast<T*>(p.out) + (bh * n + i0 + 2 * t) * kC + 4 * g;
            if (kind == kRecRuns) {
                float acc[2][2][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = acc[1][0][i] = acc[1][1][i] = 0.f;
                PairAt at[2] = {};
                if (SHIFT) {
                    at[0] = pair_at(Ah + (long long)g * p.a_row, t);
                    at[1] = pair_at(Ah + (long long)(g + 8) * p.a_row, t);
                }
                sum_head<Pick<true, false, TAIL>, T, SHIFT, 2, Tile::kSet>(at_row(Xh, 2 * t), p.x_row, w, at, sm.rec.map[g], sm, sm.tok, U0, p.pad_cl, n, t, acc);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (8 * e + 2 * t < rows) st4(o + 8 * e * kC, acc_channels(acc[e], 0));
                    if (8 * e + 2 * t + 1 < rows) st4(o + (8 * e + 1) * kC, acc_channels(acc[e], 1));
                }
            } else {
                for (int e = 0; 8 * e < rows; ++e) {
                    float acc[1][2][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = 0.f;
                    PairAt at[1] = {};
                    if (SHIFT) at[0] = pair_at(Ah + (long long)(g + 8 * e) * p.a_row, t);
                    const T* we = w + e * Tile::kSet;
                    const unsigned char* map = sm.rec.map[g + 8 * e];
                    if (kind == kRecSame) {
                        const unsigned short* tok = sm.tok + e * kGroupMaxM;
                        if (holes) sum_head<Pick<false, true>, T, SHIFT, 1, Tile::kSet>(Xh, p.x_row, we, at, map, sm, tok, U0, -1, n, t, acc);
                        else sum_head<Pick<false, false>, T, SHIFT, 1, Tile::kSet>(kF32 ? Xh - 4 * g + rows_channel<T>(lane) : Xh, p.x_row, we, at, map, sm, tok, U0, -1, n, t, acc);
                    } else if constexpr (!kF32) {
                        for (int first = 8 * e, U; first < min(rows, 8 * e + 8);) {
                            first += load_piece<RT>(src, first, rows, m, n, p.wide_idx != 0, sm, lane, &U);
                            sum_head<Pick<false, true>, T, SHIFT, 1, Tile::kSet>(Xh, p.x_row, we, at, map, sm, sm.tok, U, -1, n, t, acc);
                        }
                    }
                    if (8 * e + 2 * t < rows) st4(o + 8 * e * kC, acc_channels(acc[0], 0));
                    if (8 * e + 2 * t + 1 < rows) st4(o + (8 * e + 1) * kC, acc_channels(acc[0], 1));
                }
            }
        } else {
            using Row = std::conditional_t<kF32, SplitRow, uint4>;
            auto load_row = [&](Row& q, int row) {
                const T* y = Ah + (long long)row * p.a_row + (kF32 ? 4 : 8) * t;
                if constexpr (kF32) {
                    load_split(q, y, row < rows);
                } else {
                    q = make_uint4(0u, 0u, 0u, 0u);
                    if (row < rows) q = __ldg(reinterpret_cast<const uint4*>(y));
                }
            };
            __syncwarp();                                    // the tile is free again
            constexpr bool LIN = SHIFT;
            auto out_rows = [&]() { return static_cast<T*>(p.out) + (bh * n + i0) * m; };
            LinearRows lin = {0, 0};
            T* lt = tile;
            if (LIN) {
                lt += (reinterpret_cast<uintptr_t>(out_rows()) & 15) / sizeof(T);
                lin = {m, kF32 ? m - g : m - 2 * t};
            }
            T* at0 = LIN ? (kF32 ? lt + 2 * t * m + g : lt + g * m + 2 * t) : (kF32 ? tile + 16 * t + g : tile + g * 8 + 2 * t);
            if (kind == kRecRuns) {
                Row q[2];
                load_row(q[0], g);
                load_row(q[1], g + 8);
                if constexpr (kF32)
                    dot_head32<Pick<true, false, TAIL>, 2, Tile::kSet, LIN>(q, at_row(Xh, g), p.x_row, at0, sm.rec.map[2 * t], sm, sm.tok, U0, p.pad_cl, n, g, lin);
                else
                    dot_head16<Pick<true, false, TAIL>, T, 2, Tile::kSet, LIN>(q, at_row(Xh, g), p.x_row, at0, sm.rec.map[g], sm, sm.tok, U0, p.pad_cl, n, g, lin);
            } else {
                for (int e = 0; 8 * e < rows; ++e) {
                    Row q[1];
                    load_row(q[0], 8 * e + g);
                    auto one = [&](auto pick, const unsigned short* tok, int U) {
                        T* te = at0 + (LIN ? 8 * e * m : e * Tile::kSet);
                        if constexpr (kF32)
                            dot_head32<decltype(pick), 1, Tile::kSet, LIN>(q, Xh, p.x_row, te, sm.rec.map[8 * e + 2 * t], sm, tok, U, -1, n, g, lin);
                        else
                            dot_head16<decltype(pick), T, 1, Tile::kSet, LIN>(q, Xh, p.x_row, te, sm.rec.map[8 * e + g], sm, tok, U, -1, n, g, lin);
                    };
                    if (kind == kRecSame) {
                        if (holes) one(Pick<false, true>{}, sm.tok + e * kGroupMaxM, U0);
                        else one(Pick<false, false>{}, sm.tok + e * kGroupMaxM, U0);
                    } else {
                        for (int first = 8 * e, U; first < min(rows, 8 * e + 8);) {
                            first += load_piece<RT>(src, first, rows, m, n, p.wide_idx != 0, sm, lane, &U);
                            one(Pick<false, true>{}, sm.tok, U);
                        }
                    }
                }
            }
            __syncwarp();
            store_rows<T, RT, LIN>(LIN ? lt : tile, out_rows(), rows, m, p.R, lane);
        }
    }
}

// ----------------------------------------------------------------------------- blocks of 64 rows, 16-bit
// A CTA's four tiles are consecutive.  When all of them have whole clusters, the distinct ones among them -- 25 where the tiles by themselves
// have 4 x 13 -- go to shared memory once per head, and the products read them there (sum: ldmatrix.trans, dot: 16-byte loads).  Against
// tiles that read their own rows from L1 / L2, over records: b128 h2 n3136 bf16 dot 70 -> 61 us, sum of the model's views 88 -> 70,
// b32 h8 n1843 52 -> 39, 65 -> 45.  What is left is waiting: with its clusters on the way a block has nothing else to do, and six of them
// share an SM (issue slots 45 and 57 % busy, L1 68 and 58 %, DRAM 42 % of its rate).
constexpr int kBlockClusters = 40;               // with more of them (35 were the most in tables of 196 to 9216 tokens) each tile reads its own
constexpr int kBlockBytes = kBlockClusters * 512;

// Scores of a tile, 16 rows of 6 pieces of 8.  The pitch is an odd number of pieces, so that 8 rows' pieces of one place lie in different
// banks.  Behind them 8 pieces for the scores that nobody names.
constexpr int kBlockR = kMmax / 8;
constexpr int kScorePitch = 16 * (kBlockR + 1), kScoreNone = kTR * kScorePitch, kScoreBytes = kScoreNone + 8 * 16;
// One head, whole clusters.  xs: the block's rows (sm.rec.cl: places of the clusters there);  w, at, map: as for sum_head
template <typename T, bool SHIFT, int SET>
__device__ __forceinline__ void sum_runs(unsigned xs, const T* w, const PairAt (&at)[2], const unsigned char* map, const GroupSmem& sm, int U, int lane,
                                         float (&acc)[2][2][4]) {
    // rows of the operand: slots lane % 8 of group u (lanes 0-15) and u + 1, piece (lane / 8) % 2 and that + 2
    const unsigned a0 = xs + row_piece(lane & 7, (lane >> 3) & 1), a1 = xs + row_piece(lane & 7, ((lane >> 3) & 1) + 2);
    const unsigned short* cl = sm.rec.cl + (lane >> 4);
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 4) {
        unsigned rm[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) rm[e] = *reinterpret_cast<const unsigned*>(map + 8 * e * kMaxU + u0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && u0 + 2 >= U) break;
            const unsigned at_x = 512u * cl[u0 + 2 * h];
            unsigned a[2][4];
            ldmatrix_x4_trans(a[0], a0 + at_x);
            ldmatrix_x4_trans(a[1], a1 + at_x);
            auto weights = [&](int e, int i) -> unsigned {
                const unsigned place = byte_of(rm[e], 2 * h + i);
                const T* p = w + e * SET + 64 * place;
                if (!SHIFT) return *reinterpret_cast<const unsigned*>(p);
                const unsigned q = __funnelshift_r(*reinterpret_cast<const unsigned*>(p + at[e].first), *reinterpret_cast<const unsigned*>(p + at[e].second), at[e].bits);
                return place == 0u ? 0u : q;
            };
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const unsigned b[2] = {weights(e, 0), weights(e, 1)};
                mma16(acc[e][0], a[0], b, static_cast<const T*>(nullptr));
                mma16(acc[e][1], a[1], b, static_cast<const T*>(nullptr));
            }
        }
    }
}
// q: rows g, g + 8, channels 8t .. 8t+7.  A record's places are row addresses for stmatrix: one instruction leaves the scores of both sets of rows
// for two groups; a lane has row lane % 16 and the groups u + lane / 16
template <typename T>
__device__ __forceinline__ void dot_runs(const uint4 (&q)[2], unsigned xs, unsigned tile, const GroupSmem& sm, int U, int lane) {
    const unsigned a0[4] = {q[0].x, q[1].x, q[0].y, q[1].y}, a1[4] = {q[0].z, q[1].z, q[0].w, q[1].w};
    const T* type = nullptr;
    const unsigned row = tile + (lane & 15) * kScorePitch - 16, none = tile + kScoreNone + 16 * (lane & 7);
    const unsigned char* map = sm.rec.map[lane & 15];
    xs += row_piece(lane >> 2, lane & 3);
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 4) {
        const uint2 cl = *reinterpret_cast<const uint2*>(sm.rec.cl + u0);
        const unsigned places = *reinterpret_cast<const unsigned*>(map + u0) >> (8 * (lane >> 4));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && u0 + 2 >= U) break;
            const unsigned cc = h ? cl.y : cl.x, place = byte_of(places, 2 * h);
            const uint4 k[2] = {lds128(xs + 512u * (cc & 0xffffu)), lds128(xs + 512u * (cc >> 16))};
            float d[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned b0[2] = {k[i].x, k[i].y}, b1[2] = {k[i].z, k[i].w};
                mma16_first(d[i], a0, b0, type);
                mma16(d[i], a1, b1, type);
            }
            stmatrix_x4(place ? row + 16 * place : none, pack2(d[0][0], d[0][1], type), pack2(d[0][2], d[0][3], type), pack2(d[1][0], d[1][1], type),
                        pack2(d[1][2], d[1][3], type));
        }
    }
}

// A list of 48 rows, no slot absent, 16-bit: all but its last two groups on their way at once.  In blocks fewer warps share an SM, with less L1, than by
// tiles, and sum_head, two groups at a time, fell behind there: sum over records, tables shared by a cluster, b128 h2 n3136 bf16 68 us by
// tiles, 77 in blocks, 64 so, b32 h8 n1843 39, 50, 41, b128 h8 n196 19.1, 21.8, 19.5.  (With another two groups in flight in the same way, runs and
// rows of their own spill and take as long or longer.)  x: the head's rows at channel 4g;  tok: the list;  w, at: as for sum_head;  rows
// that do not exist take what lies in the tile, and are not stored
template <typename T, bool SHIFT>
__device__ __forceinline__ void sum_list(const T* __restrict__ x, unsigned x_row, const T* w, const PairAt& at, const unsigned short* tok, int t,
                                         float (&acc)[2][4]) {
    const unsigned* toks = reinterpret_cast<const unsigned*>(tok) + t;
    uint2 v[2][4];
    auto load = [&](int u, uint2 (&d)[4]) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned tk = toks[(u + i) * 4];
            d[2 * i] = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(x) + (unsigned long long)(tk & 0xffffu) * x_row));
            d[2 * i + 1] = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(x) + (unsigned long long)(tk >> 16) * x_row));
        }
    };
    load(0, v[0]);
    load(2, v[1]);
    cp_async_wait<0>();                                      // (the weights)
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kBlockR; u += 2) {
        uint2 (&d)[4] = v[(u >> 1) & 1];
        unsigned a[2][4], b[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const T* q = w + 64 * (u + i + 1);
            if (SHIFT) b[i] = __funnelshift_r(*reinterpret_cast<const unsigned*>(q + at.first), *reinterpret_cast<const unsigned*>(q + at.second), at.bits);
            else b[i] = *reinterpret_cast<const unsigned*>(q);
        }
        frag_channels16(a, d[0], d[1], d[2], d[3]);
        if (u + 4 < kBlockR) load(u + 4, d);
        mma16(acc[0], a[0], b, static_cast<const T*>(nullptr));
        mma16(acc[1], a[1], b, static_cast<const T*>(nullptr));
    }
}

// A tile by itself, 16-bit, its record unpacked (the weights of the first head are on their way): as in gather_groups_kernel, which has a body of its own,
// because the compiler schedules one that serves both kernels worse (fp32 dot b128 h2 n3136 174 -> 185 us, bf16 sum b64 h2 n3136 m40 41 -> 44).
// What changes in one of them changes in the other: the tests compare the two bit by bit
template <typename T, int MODE, bool SHIFT, bool TAIL>
__device__ __forceinline__ void gather_tile(const GatherGroupsParams& p, GroupSmem& sm, T* tile, const T* A, const T* X, const int64_t* src, int b, int i0, int rows,
                                            int h0, int h1, int lane) {
    using Tile = RowTile<T, kBlockR, SHIFT>;
    constexpr int m = kMmax;
    const int n = p.n;
    const int g = lane >> 2, t = lane & 3;
    const unsigned head = sm.rec.head;
    const unsigned kind = head & 0xffu;
    const bool holes = (head >> 16 & (MODE == 1 ? 1u : 3u)) != 0u;
    const int U0 = (head >> 8) & 0xffu;
    auto at_row = [&](const T* x, int row) { return reinterpret_cast<const T*>(reinterpret_cast<const char*>(x) + (unsigned long long)row * p.x_row); };
    for (int h = h0; h < h1; ++h) {
        const long long bh = (long long)b * p.heads + h;
        const T* Ah = A + (long long)h * p.a_head;
        const T* Xh = X + (long long)h * p.x_head;
        if constexpr (MODE == 0) {
            if (h > h0) {                                    // (the first head's weights were requested above)
                __syncwarp();
                stage_rows<T, kBlockR, SHIFT>(Ah, p.a_row, rows, m, kBlockR, tile, lane);
            }
            const T* w = tile + g * 8 + (SHIFT ? 0 : 2 * t);
            T* o = static_cast<T*>(p.out) + (bh * n + i0 + 2 * t) * kC + 4 * g;
            if (kind == kRecRuns) {
                float acc[2][2][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = acc[1][0][i] = acc[1][1][i] = 0.f;
                PairAt at[2] = {};
                if (SHIFT) {
                    at[0] = pair_at(Ah + (long long)g * p.a_row, t);
                    at[1] = pair_at(Ah + (long long)(g + 8) * p.a_row, t);
                }
                sum_head<Pick<true, false, TAIL>, T, SHIFT, 2, Tile::kSet>(at_row(Xh, 2 * t), p.x_row, w, at, sm.rec.map[g], sm, sm.tok, U0, p.pad_cl, n, t, acc);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (8 * e + 2 * t < rows) st4(o + 8 * e * kC, acc_channels(acc[e], 0));
                    if (8 * e + 2 * t + 1 < rows) st4(o + (8 * e + 1) * kC, acc_channels(acc[e], 1));
                }
            } else {
                for (int e = 0; 8 * e < rows; ++e) {
                    float acc[1][2][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = 0.f;
                    PairAt at[1] = {};
                    if (SHIFT) at[0] = pair_at(Ah + (long long)(g + 8 * e) * p.a_row, t);
                    const T* we = w + e * Tile::kSet;
                    const unsigned char* map = sm.rec.map[g + 8 * e];
                    if (kind == kRecSame) {
                        const unsigned short* tok = sm.tok + e * kGroupMaxM;
                        if (holes) sum_head<Pick<false, true>, T, SHIFT, 1, Tile::kSet>(Xh, p.x_row, we, at, map, sm, tok, U0, -1, n, t, acc);
                        else sum_list<T, SHIFT>(Xh, p.x_row, we, at[0], tok, t, acc[0]);
                    } else {
                        for (int first = 8 * e, U; first < min(rows, 8 * e + 8);) {
                            first += load_piece<kBlockR>(src, first, rows, m, n, p.wide_idx != 0, sm, lane, &U);
                            sum_head<Pick<false, true>, T, SHIFT, 1, Tile::kSet>(Xh, p.x_row, we, at, map, sm, sm.tok, U, -1, n, t, acc);
                        }
                    }
                    if (8 * e + 2 * t < rows) st4(o + 8 * e * kC, acc_channels(acc[0], 0));
                    if (8 * e + 2 * t + 1 < rows) st4(o + (8 * e + 1) * kC, acc_channels(acc[0], 1));
                }
            }
        } else {
            auto load_row = [&](uint4& q, int row) {
                q = make_uint4(0u, 0u, 0u, 0u);
                if (row < rows) q = __ldg(reinterpret_cast<const uint4*>(Ah + (long long)row * p.a_row + 8 * t));
            };
            __syncwarp();                                    // the tile is free again
            auto out_rows = [&]() { return static_cast<T*>(p.out) + (bh * n + i0) * m; };
            const LinearRows lin = {0, 0};
            T* at0 = tile + g * 8 + 2 * t;
            if (kind == kRecRuns) {
                uint4 q[2];
                load_row(q[0], g);
                load_row(q[1], g + 8);
                dot_head16<Pick<true, false, TAIL>, T, 2, Tile::kSet, false>(q, at_row(Xh, g), p.x_row, at0, sm.rec.map[g], sm, sm.tok, U0, p.pad_cl, n, g, lin);
            } else {
                for (int e = 0; 8 * e < rows; ++e) {
                    uint4 q[1];
                    load_row(q[0], 8 * e + g);
                    auto one = [&](auto pick, const unsigned short* tok, int U) {
                        dot_head16<decltype(pick), T, 1, Tile::kSet, false>(q, Xh, p.x_row, at0 + e * Tile::kSet, sm.rec.map[8 * e + g], sm, tok, U, -1, n, g, lin);
                    };
                    if (kind == kRecSame) {
                        if (holes) one(Pick<false, true>{}, sm.tok + e * kGroupMaxM, U0);
                        else one(Pick<false, false>{}, sm.tok + e * kGroupMaxM, U0);
                    } else {
                        for (int first = 8 * e, U; first < min(rows, 8 * e + 8);) {
                            first += load_piece<kBlockR>(src, first, rows, m, n, p.wide_idx != 0, sm, lane, &U);
                            one(Pick<false, true>{}, sm.tok, U);
                        }
                    }
                }
            }
            __syncwarp();
            store_rows<T, kBlockR, false>(tile, out_rows(), rows, m, kBlockR, lane);
        }
    }
}

template <typename T, int MODE, bool SHIFT, bool TAIL>
__global__ void __launch_bounds__(32 * kGWarps, kBlockCtas)
gather_blocks_kernel(const __grid_constant__ GatherGroupsParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned short block_cl[kBlockClusters];
    __shared__ int block_count;
    using Tile = RowTile<T, kBlockR, SHIFT>;
    constexpr int kTile = MODE == 1 ? kScoreBytes : Tile::kBytes;
    static_assert(kTile >= Tile::kBytes, "a tile by itself has its place");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* base = smem_raw + warp * (int)(sizeof(GroupSmem) + kTile);
    unsigned char* xbuf = smem_raw + kGWarps * (int)(sizeof(GroupSmem) + kTile);
    GroupSmem& sm = *reinterpret_cast<GroupSmem*>(base);
    T* tile = reinterpret_cast<T*>(base + sizeof(GroupSmem));
    const unsigned blocks = (unsigned)(p.tiles + kGWarps - 1) / kGWarps, bb = blockIdx.x / (unsigned)p.parts;
    const int part = (int)(blockIdx.x - bb * (unsigned)p.parts);
    const int b = (int)(bb / blocks);
    const int ti = (int)(bb - (unsigned)b * blocks) * kGWarps + warp;
    const bool live = ti < p.tiles;
    const int i0 = ti * kTR;
    constexpr int m = kMmax;
    const int n = p.n;
    const int rows = live ? min(kTR, n - i0) : 0;
    const int g = lane >> 2, t = lane & 3;
    const int h0 = part * p.per_part, h1 = min(p.heads, h0 + p.per_part);
    const T* A = static_cast<const T*>(p.A) + (long long)b * p.a_batch + (long long)i0 * p.a_row;
    const int64_t* src = p.idx + ((long long)b * n + i0) * m;
    const unsigned tile_s = smem_u32(tile);
    if (live) {
        reinterpret_cast<uint4*>(&sm.rec)[lane] = __ldg(reinterpret_cast<const uint4*>(p.plan + (long long)b * p.tiles + ti) + lane);
        __syncwarp();
        if (MODE == 0) {
            if (!SHIFT) {                                    // the zeros of place 0
                for (int z = lane; z < 2 * Tile::kPlace * (int)sizeof(T) / 16; z += 32) {
                    constexpr int kPer = 16 / (int)sizeof(T);
                    const int e = z / (Tile::kPlace / kPer), c = z % (Tile::kPlace / kPer);
                    *reinterpret_cast<uint4*>(tile + e * Tile::kSet + c * kPer) = make_uint4(0u, 0u, 0u, 0u);
                }
            }
            stage_rows<T, kBlockR, SHIFT>(A + (long long)h0 * p.a_head, p.a_row, rows, m, kBlockR, tile, lane);
        }
    }
    if (__syncthreads_and(!live || (sm.rec.head & 0xffu) == kRecRuns)) {
        // ---- the distinct clusters of the block: a bit each, their places by population count
        unsigned* bits = reinterpret_cast<unsigned*>(xbuf);
        unsigned short* before = reinterpret_cast<unsigned short*>(xbuf + 1024);
        const int words = (n + 255) >> 8;                    // (at most 254)
        for (int z = threadIdx.x; z < words; z += 32 * kGWarps) bits[z] = 0u;
        __syncthreads();
        const int U = live ? (int)(sm.rec.head >> 8 & 0xffu) : 0;
        const unsigned cl = lane < U ? sm.rec.cl[lane] : 0u;
        if (lane < U) atomicOr(&bits[cl >> 5], 1u << (cl & 31u));
        __syncthreads();
        if (warp == 0) {
            int run = 0;
            for (int z = 0; z < words; z += 32) {
                const int v = z + lane < words ? __popc(bits[z + lane]) : 0;
                int incl = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += y;
                }
                if (z + lane < words) before[z + lane] = (unsigned short)(run + incl - v);
                run += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0) block_count = run;
        }
        __syncthreads();
        const int total = block_count;
        if (total <= kBlockClusters) {
            const unsigned place = before[cl >> 5] + __popc(bits[cl >> 5] & ((1u << (cl & 31u)) - 1u));
            const unsigned place0 = __shfl_sync(kFull, place, 0);
            if (lane < U) {
                sm.rec.cl[lane] = (unsigned short)place;
                block_cl[place] = (unsigned short)cl;
            } else if (lane == U && (U & 1)) {
                sm.rec.cl[U] = (unsigned short)place0;
            }
            const unsigned xs = smem_u32(xbuf), x_dst = xs + 512u * warp + row_piece(g, t);
            const char* xh = static_cast<const char*>(p.X) + 2 * ((long long)b * p.x_batch + (long long)h0 * p.x_head) + (unsigned long long)g * p.x_row + 16 * t;
            const T* Ah = A + (long long)h0 * p.a_head;
            long long bh = (long long)b * p.heads + h0;
            for (int h = h0; h < h1; ++h, xh += 2 * p.x_head, Ah += p.a_head, ++bh) {
                __syncthreads();                             // the clusters of the head before, or the bits, are done with
                unsigned dst = x_dst;
#pragma unroll 2
                for (int u = warp; u < total; u += kGWarps, dst += 512u * kGWarps) {
                    const unsigned first = 8u * block_cl[u];
                    const char* from = xh + (unsigned long long)first * p.x_row;
                    if (TAIL && first + g >= (unsigned)n) from = xh - (unsigned long long)g * p.x_row;      // slots behind the last token: token 0
                    cp_async16_cg(dst, from);
                }
                if (MODE == 0 && h > h0 && live) stage_rows<T, kBlockR, SHIFT>(Ah, p.a_row, rows, m, kBlockR, tile, lane);
                cp_async_commit();
                if constexpr (MODE == 0) {
                    cp_async_wait<0>();
                    __syncthreads();
                    if (!live) continue;
                    float acc[2][2][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[0][0][i] = acc[0][1][i] = acc[1][0][i] = acc[1][1][i] = 0.f;
                    PairAt at[2] = {};
                    if (SHIFT) {
                        at[0] = pair_at(Ah + (long long)g * p.a_row, t);
                        at[1] = pair_at(Ah + (long long)(g + 8) * p.a_row, t);
                    }
                    sum_runs<T, SHIFT, Tile::kSet>(xs, tile + g * 8 + (SHIFT ? 0 : 2 * t), at, sm.rec.map[g], sm, U, lane, acc);
                    const unsigned buf = smem_u32(sm.tok);
                    T* o = static_cast<T*>(p.out) + (bh * n + i0 + g) * kC + 8 * t;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        __syncwarp();
                        acc_to_rows<T>(acc[e], buf, lane);
                        __syncwarp();
                        if (8 * e + g < rows) *reinterpret_cast<uint4*>(o + 8 * e * kC) = lds128(buf + row_piece(g, t));
                    }
                } else {
                    uint4 q[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        q[e] = make_uint4(0u, 0u, 0u, 0u);
                        if (8 * e + g < rows) q[e] = __ldg(reinterpret_cast<const uint4*>(Ah + (long long)(8 * e + g) * p.a_row + 8 * t));
                    }
                    cp_async_wait<0>();
                    __syncthreads();
                    if (!live) continue;
                    dot_runs<T>(q, xs, tile_s, sm, U, lane);
                    __syncwarp();
                    T* o = static_cast<T*>(p.out) + (bh * n + i0) * m;
#pragma unroll
                    for (int k = 0; k < kBlockR / 2; ++k) {
                        const int z = lane + 32 * k, row = z / kBlockR, j = z - row * kBlockR;
                        if (row < rows) *reinterpret_cast<uint4*>(o + 8 * z) = lds128(tile_s + row * kScorePitch + 16 * j);
                    }
                }
            }
            return;
        }
    }
    if (!live) return;
    unpack_record<MODE == 1>(sm, rows, lane);
    gather_tile<T, MODE, SHIFT, TAIL>(p, sm, tile, A, static_cast<const T*>(p.X) + (long long)b * p.x_batch + (MODE == 0 ? 4 * g : 8 * t), src, b, i0, rows,
                                          h0, h1, lane);
}

template <typename T, int MODE>
int gather_groups_t(const char* label, GatherGroupsParams p, int b, cudaStream_t s) {
    p.tiles = group_tiles(p.n);
    p.R = (p.m + 7) / 8;
    const long long tiles = (long long)b * p.tiles;
    if (tiles * p.heads > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    p.wide_idx = p.m % 8 == 0 && reinterpret_cast<uintptr_t>(p.idx) % 16 == 0;
    const bool m48 = p.m == kMmax && p.wide_idx;
    // 16-bit tiles share their rows in blocks over records.  Where the records are made here, most of the time goes there: sum b128 h2 n3136 bf16
    // 94 us, 92 in blocks, but for tables shared by a cluster 84, 97;  dot 92, 97.  Other rows than of 48 have records in the forward passes too,
    // where shared tables lose as well (b64 h8 n784 m24 dot 37 us, 44 in blocks).  Which kind a table is, the host does not know: what blocks
    // cannot serve goes tile by tile inside, and is slower there than in the kernel of tiles where rows have little in common (sum by tiles / here:
    // tiles in any order, blocks of more than 40 clusters, b128 h2 n3136 80 / 89; random rows b32 h8 n1843 229 / 260, b4 h4 n784 19.5 / 20.2).
    // Dot products only from 128 (tile, head) pairs per SM on: a block has barriers, and its clusters on the way, in front of few products (QK forward over records,
    // us by tiles / in blocks: b128 h8 n196 16.8 / 17.4, b16 h2 n3136 10.3 / 11.3, b4 h2 n9216 8.1 / 10.1, b4 h4 n784 4.4 / 4.8; above:
    // b64 h8 n784 33 / 30, b32 h8 n1843 52 / 39).  Sums gain at every size (b128 h8 n196 22 / 19, b4 h2 n9216 11.8 / 10.9, b1 h8 n196 5.0 / 4.3).
    constexpr bool kBlocks = sizeof(T) == 2;
    const bool blocks = kBlocks && p.plan && m48 && (MODE == 0 || tiles * p.heads >= 128LL * sm_count());
    // (a block does little before its first head, and is large: b32 h8 n1843 44 -> 39 us (dot), 47 -> 41 (sum) with 40 warps per SM instead of 24,
    // b128 h8 n196 sum 18.8 with both; 20.9 with 64)
    split_heads(tiles, p.heads, &p.parts, &p.per_part, blocks ? 40 : 24);
    p.total = (unsigned)(tiles * p.parts);
    p.pad_cl = p.n % 8 ? p.n / 8 : -1;
    constexpr int kPer = 16 / (int)sizeof(T);
    const bool shift = p.m % 8 != 0 || (MODE == 0 && !(reinterpret_cast<uintptr_t>(p.A) % 16 == 0 && p.a_row % kPer == 0 && p.a_batch % kPer == 0 &&
                                                       p.a_head % kPer == 0));
    auto pick = [&](auto plan, auto tail) {
        constexpr bool PLAN = decltype(plan)::value, TAIL = decltype(tail)::value;
        if constexpr (kBlocks && PLAN) {
            if (blocks) return shift ? gather_blocks_kernel<T, MODE, MODE == 0, TAIL> : gather_blocks_kernel<T, MODE, false, TAIL>;
            if constexpr (MODE == 0) return shift ? gather_groups_kernel<T, MODE, 0, true, PLAN, true> : gather_groups_kernel<T, MODE, 0, false, PLAN, true>;
        }
        return m48 ? (shift ? gather_groups_kernel<T, MODE, 6, MODE == 0, PLAN, TAIL> : gather_groups_kernel<T, MODE, 6, false, PLAN, TAIL>)
                   : (shift ? gather_groups_kernel<T, MODE, 0, true, PLAN, true> : gather_groups_kernel<T, MODE, 0, false, PLAN, true>);
    };
    auto kernel = p.plan ? (p.pad_cl >= 0 ? pick(std::true_type{}, std::true_type{}) : pick(std::true_type{}, std::false_type{}))
                         : (p.pad_cl >= 0 ? pick(std::false_type{}, std::true_type{}) : pick(std::false_type{}, std::false_type{}));
    const int rows_tile = m48 ? (shift ? RowTile<T, 6, true>::kBytes : RowTile<T, 6, false>::kBytes)
                              : (shift ? RowTile<T, 0, true>::kBytes : RowTile<T, 0, false>::kBytes);
    const int smem = kGWarps * ((int)sizeof(GroupSmem) + (blocks && MODE == 1 ? kScoreBytes : rows_tile)) + (blocks ? kBlockBytes : 0);
    const unsigned grid = blocks ? (unsigned)(b * ((p.tiles + kGWarps - 1) / kGWarps) * p.parts) : (p.total + kGWarps - 1) / kGWarps;
    const int fit = resident_ctas(reinterpret_cast<const void*>(kernel), 32 * kGWarps, smem);
    if (fit < 0) return fit;
    ScopedKernelTimer timer(label, s);
    kernel<<<grid, 32 * kGWarps, smem, s>>>(p);
    note_launch();
    return check_launch();
}

bool gather_supported(int dtype, std::initializer_list<const void*> ptrs, int n, int m, int c) {
    if (c != kC || m < 1 || m > kGroupMaxM || n < 1 || n > 65000) return false;
    // fp32 rows of more than 48: the plain FMAs of generic.cu, whose error against 64 bits is 1.0e-7 .. 1.4e-7 where three TF32 passes
    // have 4.6e-7 .. 7.8e-7 (2-norm, n49 m49 .. n64 m64).  They are slower: b256 h16 n49 m49 350 / 292 us for QK / AV against 88 / 78.
    if (dtype == CLUSTEN_F32 && m > kMmax) return false;
    if (dtype != CLUSTEN_F32 && dtype != CLUSTEN_F16 && dtype != CLUSTEN_BF16) return false;
    for (const void* p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
    return true;
}

GatherGroupsParams gather_params(const void* A, const void* X, const int64_t* idx, void* out, int h, int n, int m, int a_cols,
                                 unsigned esize, const GatherStrides& gs,
                                 const void* plan) {
    GatherGroupsParams p{};
    p.A = A;  p.X = X;  p.idx = idx;  p.out = out;
    p.heads = h;  p.n = n;  p.m = m;
    p.a_batch = (long long)h * n * a_cols;  p.a_head = (long long)n * a_cols;  p.a_row = a_cols;
    p.x_batch = (long long)h * n * kC;  p.x_head = (long long)n * kC;  p.x_row = kC;
    if (gs.y_row != 0) {
        p.a_batch = gs.y_batch;  p.a_head = gs.y_head;  p.a_row = (int)gs.y_row;
    }
    if (gs.x_row != 0) {
        p.x_batch = gs.x_batch;  p.x_head = gs.x_head;  p.x_row = (unsigned)gs.x_row;
    }
    p.x_row *= esize;
    p.plan = static_cast<const TileRecord*>(plan);
    return p;
}

}  // namespace

bool tiled_sum_supported(int dtype, const void* W, const void* X, const void* out, int n, int m, int c) {
    return gather_supported(dtype, {X, out}, n, m, c) && W != nullptr;
}
int launch_tiled_sum(const char* label, int dtype, const void* W, const void* X, const int64_t* idx, void* out,
                     int b, int h, int n, int m, cudaStream_t s, const GatherStrides& gs, const void* plan) {
    const GatherGroupsParams p = gather_params(W, X, idx, out, h, n, m, m, dtype_size(dtype), gs, plan);
    switch (dtype) {
        case CLUSTEN_F32: return gather_groups_t<float, 0>(label, p, b, s);
        case CLUSTEN_F16: return gather_groups_t<__half, 0>(label, p, b, s);
        case CLUSTEN_BF16: return gather_groups_t<__nv_bfloat16, 0>(label, p, b, s);
        default: return CLUSTEN_ERR_DTYPE;
    }
}

bool tiled_dot_supported(int dtype, const void* Y, const void* X, const void* out, int n, int m, int c) {
    return gather_supported(dtype, {Y, X, out}, n, m, c);
}
int launch_tiled_dot(const char* label, int dtype, const void* X, const void* Y, const int64_t* idx, void* out,
                     int b, int h, int n, int m, cudaStream_t s, const GatherStrides& gs, const void* plan) {
    const GatherGroupsParams p = gather_params(Y, X, idx, out, h, n, m, kC, dtype_size(dtype), gs, plan);
    switch (dtype) {
        case CLUSTEN_F32: return gather_groups_t<float, 1>(label, p, b, s);
        case CLUSTEN_F16: return gather_groups_t<__half, 1>(label, p, b, s);
        case CLUSTEN_BF16: return gather_groups_t<__nv_bfloat16, 1>(label, p, b, s);
        default: return CLUSTEN_ERR_DTYPE;
    }
}

}  // namespace clusten
