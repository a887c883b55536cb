// Building blocks of the kernels that work on GROUPS of 8 neighbour slots (gather_groups.cu, fused_attn.cu).
//
// A warp owns a tile of 16 consecutive rows of one batch element.  Lane (g, t) = (lane / 4, lane % 4) owns the rows g
// and g + 8 and, of every group of 8 slots 8r .. 8r+7, the slots 8r + 2t and 8r + 2t + 1 -- the element layout that
// mma.sync gives its A operand's rows, its accumulator and the columns of its B operand, so that neighbour rows go
// from L1 / L2 straight into operand registers: no staging, no transposition.
//
// The kernels' currencies are instructions and L1 wavefronts (one per distinct 128-byte line of a request).  Hence
//   * the neighbours of the 16 rows are merged, so that a neighbour row is read once per tile (12.9 distinct groups per
//     16 rows of an AutoFocusFormer stage against 2 x 10.2 for two tiles of 8);
//   * everything that is contiguous per tile (indices, weights, scores) is read and written contiguously;
//   * the list of a tile's groups is a RECORD of 512 bytes that one kernel writes once per table (group_plan.cu) and
//     every consumer reads with one 16-byte load per lane, instead of 6 KB of int64 indices and their analysis.
//
// A record is of one of three kinds:
//   runs    every group of every row is one cluster of 8 consecutive tokens 8c .. 8c+7 (the last cluster padded with
//           token 0), which is what AutoFocusFormer builds (models/aff_transformer.py:476-482 of the reference): the
//           distinct clusters, and per row and cluster its place among the row's groups
//   same    rows 0 .. 7 are one list and so are rows 8 .. 15 (tables shared by the tokens of a cluster): the two lists
//   other   anything else: the consumer reads the indices itself, a few rows at a time (load_piece)
#pragma once

#include "index_arithmetic.h"
#include "tile_core.cuh"

namespace clusten {
namespace {

constexpr int kTR = 16;                          // rows per tile
constexpr int kGroupMaxR = 8;                    // groups per row: m <= 64
constexpr int kGroupMaxM = 8 * kGroupMaxR;
constexpr int kMaxU = 28;                        // distinct groups of a record or piece
constexpr int kTagSpan = 1024;                   // tags by cluster id, from the lowest one on and modulo this
constexpr unsigned kRecRuns = 0, kRecSame = 1, kRecOther = 2;

struct __align__(16) TileRecord {
    unsigned head;                               // kind | groups << 8 | some slot is absent << 16 | an odd number of groups in a list << 17
    unsigned unused;
    unsigned short cl[kMaxU];                    // runs: the clusters (behind an odd number of them the first one again)
    union {
        unsigned char map[kTR][kMaxU];           // [row][group]: place of the group in the row + 1, 0: not named by it
        unsigned short lists[2][kGroupMaxM];     // same: source rows by slot (0xffff: absent, and so are the slots behind the last group)
    };
};
static_assert(sizeof(TileRecord) == 512, "one 16-byte piece per lane");

struct __align__(16) GroupSmem {                 // one per warp
    TileRecord rec;
    unsigned short tok[8 * 32];                  // same: [list][64], other: [group][8]: source rows
};

__device__ __forceinline__ unsigned pair16(int lo, int hi) { return (unsigned)lo | ((unsigned)hi << 16); }

// ----------------------------------------------------------------------------- record of a tile, from its indices
// src = index rows of the tile (rows of them exist), n_src source rows (at most 65000).  rec, tag (kTagSpan bytes): shared
// memory of the warp.  RT: groups per row when known at compile time (m = 8 RT; 0: R_arg);  TAIL: n_src is not a
// multiple of 8;  wide: m is a multiple of 8 and the rows start on 16-byte boundaries;  DIVIDE: not by multiplication, which costs registers.
// The runs y = row * R + r are read in memory order, run y = g + 8 k by the four lanes (g, t).
template <int RT, bool TAIL, bool DIVIDE = true>
__device__ __forceinline__ void build_record(const int64_t* __restrict__ src, int rows, int m, int R_arg, int n_src, bool wide,
                                             TileRecord& rec, unsigned char* tag, int lane) {
    constexpr int RMAX = RT > 0 ? RT : kGroupMaxR;
    const int R = RT > 0 ? RT : R_arg;
    const int g = lane >> 2, t = lane & 3;
    const int nruns = rows * R;
    // y / R, exact for y < 128
    const unsigned inverse = DIVIDE ? 0u : (65536u + (unsigned)R - 1u) / (unsigned)R;
    auto row_of = [&](int y) { return DIVIDE ? y / R : (int)((unsigned)y * inverse >> 16); };
    unsigned pr[2 * RMAX];                                   // this lane's two tokens of run g + 8 k (0xffff: absent)
    unsigned out = 0u;                                       // not zero: an index out of range
    if (RT > 0 || wide) {
        const longlong2* p = reinterpret_cast<const longlong2*>(src) + lane;      // 4 pairs per run
        unsigned top = 0u;
#pragma unroll
        for (int k = 0; k < 2 * RMAX; ++k) {
            int4 v = make_int4(0, 0, 0, 0);                                       // {lo, hi, lo, hi} of two indices
            if (g + 8 * k < nruns) v = __ldg(reinterpret_cast<const int4*>(p + 32 * k));
            pr[k] = __byte_perm((unsigned)v.x, (unsigned)v.z, 0x5410);
            top = max(top, max((unsigned)v.x, (unsigned)v.z));
            out |= (unsigned)(v.y | v.w);
        }
        out |= top >= (unsigned)n_src ? 1u : 0u;
    } else {
#pragma unroll
        for (int k = 0; k < 2 * RMAX; ++k) {
            const int y = g + 8 * k;
            pr[k] = 0xffffffffu;
            if (y < nruns) {
                const int row = row_of(y), j = 8 * (y - row * R) + 2 * t;
                const int64_t* q = src + (long long)row * m + j;
                const long long a = j < m ? __ldg(q) : -1, b = j + 1 < m ? __ldg(q + 1) : -1;
                pr[k] = pair16((unsigned long long)a < (unsigned long long)n_src ? (int)a : kSkip,
                               (unsigned long long)b < (unsigned long long)n_src ? (int)b : kSkip);
            }
        }
    }
    __syncwarp();                                            // an earlier record may still be in use
    reinterpret_cast<uint4*>(&rec)[lane] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    const bool inside = !__any_sync(kFull, out != 0u);
    // ---- whole clusters?
    unsigned bad = inside && (RT > 0 || wide) ? 0u : 1u;
    unsigned f[RMAX];                                        // first tokens of the runs, two per register
    const bool spread = n_src > 8 * kTagSpan;                // uniform; else the tags cover every cluster there is
    unsigned lo = spread ? 0xffffu : 0u, hi = spread ? 0u : (unsigned)(n_src - 1);
    const unsigned mine = pair16(2 * t, 2 * t + 1);
#pragma unroll
    for (int k = 0; k < 2 * RMAX; ++k) {
        const unsigned first = __shfl_sync(kFull, pr[k], lane & 28) & 0xffffu;
        unsigned want = first * 0x10001u + mine;
        if (TAIL) {                                          // the last cluster is padded with token 0
            if ((want & 0xffffu) >= (unsigned)n_src) want = 0u;
            else if ((want >> 16) >= (unsigned)n_src) want &= 0xffffu;
        }
        if (g + 8 * k < nruns) {
            bad |= (pr[k] ^ want) | (first & 7u);
            if (spread) {
                lo = min(lo, first);
                hi = max(hi, first);
            }
        }
        if (k & 1) f[k >> 1] |= first << 16;
        else f[k >> 1] = first;
    }
    if (spread) {
        lo = __reduce_min_sync(kFull, lo);
        hi = __reduce_max_sync(kFull, hi);
    }
    lo >>= 3;
    hi >>= 3;
    if (!__any_sync(kFull, bad != 0u)) {
        // Clusters are numbered through a table of tags.  When a tile's span more ids than it has entries (the curve along which
        // tokens are numbered leaves and comes back), two of them may share a tag: a run that finds another cluster there
        // sees it in rec.cl, and the tile is not of this kind.
        const bool wide_span = hi - lo >= kTagSpan;          // uniform
        bool shared = false;
        for (int z = lane; 16 * z <= (int)min(hi - lo, (unsigned)kTagSpan - 1u); z += 32)
            reinterpret_cast<uint4*>(tag)[z] = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        __syncwarp();
        constexpr int NB = (2 * RMAX + 3) / 4;               // batches of 32 runs, one per lane: run g + 8 (4 j + t)
        unsigned slots = 0u;                                 // a byte per batch
        int U = 0;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int y = g + 8 * (4 * j + t);
            const bool live = y < nruns && (RT == 0 || 4 * j + t < 2 * RT);
            const unsigned ff = (t & 2) && 2 * j + 1 < RMAX ? f[2 * j + 1 < RMAX ? 2 * j + 1 : 0] : f[2 * j];
            const unsigned cl = ((t & 1) ? ff >> 16 : ff & 0xffffu) >> 3;
            // groups are numbered in the order in which the runs first name them
            const unsigned peers = __match_any_sync(kFull, live ? cl : 0x10000u + lane);
            const bool lead = live && (peers & ((1u << lane) - 1u)) == 0u;
            unsigned char* mytag = tag + (live ? (cl - lo) & (kTagSpan - 1) : 0u);
            const bool fresh = lead && *mytag == 0xffu;
            const unsigned nb = __ballot_sync(kFull, fresh);
            const int slot = U + __popc(nb & ((1u << lane) - 1u));
            U += __popc(nb);
            if (U > kMaxU) break;                            // uniform
            if (fresh) {
                *mytag = (unsigned char)slot;
                rec.cl[slot] = (unsigned short)cl;
            }
            __syncwarp();
            const unsigned s = live ? *mytag : 0u;
            slots |= s << (8 * j);
            if (wide_span) shared = shared || (live && rec.cl[s] != cl);
            const int row = y / R;
            if (live) rec.map[row][s] = (unsigned char)(y - row * R + 1);
        }
        __syncwarp();
        bool twice = U > kMaxU || shared;
        if (U <= kMaxU) {
            // a row that names a cluster twice has overwritten its own entry
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                const int y = g + 8 * (4 * j + t);
                const int row = y / R;
                if (y < nruns && (RT == 0 || 4 * j + t < 2 * RT)) twice = twice || rec.map[row][(slots >> (8 * j)) & 0xffu] != y - row * R + 1;
            }
        }
        if (!__any_sync(kFull, twice)) {
            if (lane == 0) {
                rec.head = kRecRuns | (unsigned)U << 8;
                // groups are taken in pairs: what is multiplied with zeros in place of one more must be the tile's own rows
                if (U & 1) rec.cl[U] = rec.cl[0];
            }
            __syncwarp();
            return;
        }
    }
    // ---- one list per 8 rows?  Run r of row 0 (8) is run y = r (8 R + r): register 0 (R), lanes (r, .)
    unsigned ref8 = pr[0];
    if (RT > 0) {
        ref8 = pr[RT];
    } else {
#pragma unroll
        for (int i = 1; i <= kGroupMaxR; ++i)
            if (i == R) ref8 = pr[i];
    }
    bool same = inside, hole = false;
#pragma unroll
    for (int k = 0; k < 2 * RMAX; ++k) {
        const int y = g + 8 * k;
        const int row = row_of(y), r = y - row * R;
        unsigned ref;
        if (RT > 0) {
            ref = __shfl_sync(kFull, k < RT ? pr[0] : ref8, 4 * r + t);
        } else {
            const unsigned ra = __shfl_sync(kFull, pr[0], 4 * r + t), rb = __shfl_sync(kFull, ref8, 4 * r + t);
            ref = row < 8 ? ra : rb;
        }
        if (y < nruns) {
            same = same && pr[k] == ref;
            hole = hole || (pr[k] & 0xffffu) == kSkip || (pr[k] >> 16) == kSkip;
        }
    }
    same = __all_sync(kFull, same);
    hole = __any_sync(kFull, hole);
    __syncwarp();
    if (same) {
        // groups are taken in pairs, so that of an odd number of them one more is looked at: absent slots (and not the places that
        // the attempt above may have left here)
        if (lane < (int)sizeof(rec.lists) / 16) reinterpret_cast<uint4*>(rec.lists)[lane] = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2 * RMAX; ++k) {
            const int y = g + 8 * k;
            const int row = row_of(y), r = y - row * R;
            if (y < nruns && (row & 7) == 0) reinterpret_cast<unsigned*>(rec.lists[row >> 3])[4 * r + t] = pr[k];
        }
    }
    if (lane == 0) rec.head = same ? (kRecSame | (unsigned)R << 8 | (hole ? 1u << 16 : 0u) | (unsigned)(R & 1) << 17) : kRecOther;
    __syncwarp();
}

// ----------------------------------------------------------------------------- groups of a tile, for its consumers
// The record in sm.rec -> what the products read.  "same": the lists move to sm.tok, and the groups of every row that exists
// (`rows` of them) are 0 .. R - 1 of its list.  FILL: the absent group behind an odd number of them repeats a token of the list, for
// consumers to whom a product that nobody looks at, or a zero weight, does no harm.
template <bool FILL>
__device__ __forceinline__ void unpack_record(GroupSmem& sm, int rows, int lane) {
    __syncwarp();
    if ((sm.rec.head & 0xffu) == kRecSame) {
        const int R = (sm.rec.head >> 8) & 0xffu;
        uint2 v = reinterpret_cast<const uint2*>(sm.rec.lists)[lane];
        if (FILL && 4 * (lane & 15) >= 8 * R) v.x = v.y = sm.rec.lists[lane >> 4][0] * 0x10001u;
        __syncwarp();
        reinterpret_cast<uint2*>(sm.tok)[lane] = v;
        for (int z = lane; z < kTR * kMaxU / 4; z += 32) {
            reinterpret_cast<unsigned*>(sm.rec.map)[z] = list_places(z / (kMaxU / 4), 4 * (z % (kMaxU / 4)), R, rows);
        }
        __syncwarp();
    }
}

// Any rows: those from `first` on, as many as fit a piece (at most to row `rows`), each with its own groups.  Returns
// the number of rows; *U their groups.  A lane reads two neighbouring slots of every row (wide: as one 16-byte load).
template <int RT>
__device__ __noinline__ int load_piece(const int64_t* __restrict__ src, int first, int rows, int m, int n_src, bool wide, GroupSmem& sm,
                                       int lane, int* U) {
    const int R = RT > 0 ? RT : (m + 7) >> 3;
    // a piece ends with its set of 8 rows
    const int take = min(min(kMaxU / R, rows - first), 8 - (first & 7));
    const int j = 2 * lane;
    const int64_t* p = src + (long long)first * m + j;
    auto token = [&](long long v) { return (unsigned long long)v < (unsigned long long)n_src ? (int)v : kSkip; };
    __syncwarp();
    for (int z = lane; z < kTR * kMaxU / 4; z += 32) reinterpret_cast<unsigned*>(sm.rec.map)[z] = 0u;
    unsigned* tok = reinterpret_cast<unsigned*>(sm.tok) + lane;
#pragma unroll 4
    for (int i = 0; i < take; ++i, p += m, tok += 4 * R) {
        longlong2 v = make_longlong2(-1, -1);
        if (RT > 0 || wide) {
            if (j < m) v = __ldg(reinterpret_cast<const longlong2*>(p));
        } else {
            if (j < m) v.x = __ldg(p);
            if (j + 1 < m) v.y = __ldg(p + 1);
        }
        if (j < 8 * R) *tok = pair16(token(v.x), token(v.y));
    }
    if (lane < 4) reinterpret_cast<unsigned*>(sm.tok)[4 * R * take + lane] = 0xffffffffu;      // (groups are taken in pairs)
    __syncwarp();
    if (lane < take * R) sm.rec.map[first + lane / R][lane] = (unsigned char)(lane % R + 1);
    __syncwarp();
    *U = take * R;
    return take;
}

// Sources of one piece of a tile.  RUNS: group u is cluster cl[u], one of them may be padded (TAIL);  else: its rows are
// tok[8 u ..], absent where HOLES.
template <bool RUNS_, bool HOLES_, bool TAIL_ = true> struct Pick {
    static constexpr bool kRuns = RUNS_, kHoles = HOLES_, kTail = TAIL_;
};

// ---- operand registers from four neighbour rows: channels 4g .. 4g+3 of every row
// 16-bit: A of m16n8k16, M tile mt = channels 4g + 2mt (row g) and 4g + 2mt + 1 (row g + 8), k = slots 2t, 2t+1 of
// group u (x0, x1) and of group u + 1 (x2, x3)
__device__ __forceinline__ void frag_channels16(unsigned (&a)[2][4], const uint2& x0, const uint2& x1, const uint2& x2, const uint2& x3) {
    a[0][0] = __byte_perm(x0.x, x1.x, 0x5410);  a[0][1] = __byte_perm(x0.x, x1.x, 0x7632);
    a[0][2] = __byte_perm(x2.x, x3.x, 0x5410);  a[0][3] = __byte_perm(x2.x, x3.x, 0x7632);
    a[1][0] = __byte_perm(x0.y, x1.y, 0x5410);  a[1][1] = __byte_perm(x0.y, x1.y, 0x7632);
    a[1][2] = __byte_perm(x2.y, x3.y, 0x5410);  a[1][3] = __byte_perm(x2.y, x3.y, 0x7632);
}
// the accumulators of the two M tiles: channels 4g .. 4g+3 of row 2t (q = 0) or 2t + 1 (q = 1)
__device__ __forceinline__ float4 acc_channels(const float (&d)[2][4], int q) {
    return q == 0 ? make_float4(d[0][0], d[0][2], d[1][0], d[1][2]) : make_float4(d[0][1], d[0][3], d[1][1], d[1][3]);
}

// two fp32 values as a 16-bit pair of the element type
__device__ __forceinline__ unsigned pack2(float lo, float hi, const __half*) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ unsigned pack2(float lo, float hi, const __nv_bfloat16*) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

// products whose accumulator starts at zero
__device__ __forceinline__ void mma16_first(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2], const __half*) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma16_first(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2], const __nv_bfloat16*) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma_tf32_first(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// mma_pair of fp32 values (tile_core.cuh) whose accumulators start at zero
__device__ __forceinline__ void mma_pair_first(float (&d)[2][4], const float (&a)[2][4], const float (&b)[2]) {
    unsigned ah[2][4], al[2][4], bh[2], bl[2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) split_tf32(a[mt][i], ah[mt][i], al[mt][i]);
#pragma unroll
    for (int i = 0; i < 2; ++i) split_tf32(b[i], bh[i], bl[i]);
    mma_tf32_first(d[0], al[0], bh);
    mma_tf32_first(d[1], al[1], bh);
    mma_tf32(d[0], ah[0], bl);
    mma_tf32(d[1], ah[1], bl);
    mma_tf32(d[0], ah[0], bh);
    mma_tf32(d[1], ah[1], bh);
}

// Four channels of a row, as the element type's vector
template <typename T> struct Four { using type = uint2; };
template <> struct Four<float> { using type = float4; };
template <typename T> using Four_t = typename Four<T>::type;
__device__ __forceinline__ void zero4(uint2& v) { v = make_uint2(0u, 0u); }
__device__ __forceinline__ void zero4(float4& v) { v = make_float4(0.f, 0.f, 0.f, 0.f); }

// Channels 4g .. 4g+3 of the slots 2t, 2t + 1 of groups u, u + 1 (u even).  x: the head's rows at channel 4g, x_row in bytes
// (RUNS: at row 2t);  pad_cl: the cluster that is padded with token 0 (-1: none), n source rows.  tk: the slots' rows, when
// not RUNS.
template <typename PICK, typename T>
__device__ __forceinline__ void load_four(Four_t<T> (&v)[4], const char* x, unsigned x_row, const GroupSmem& sm, const unsigned short* tok, int u,
                                          int t, int pad_cl, int n, unsigned (&tk)[2]) {
    using V = Four_t<T>;
    if constexpr (PICK::kRuns) {
        const unsigned cc = *reinterpret_cast<const unsigned*>(sm.rec.cl + u);
        const char* x1 = x + x_row;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned c = i == 0 ? cc & 0xffffu : cc >> 16;
            const char* p0 = x + (unsigned long long)(8u * c) * x_row;
            const char* p1 = x1 + (unsigned long long)(8u * c) * x_row;
            if (PICK::kTail) {                               // slots behind the last token: token 0
                const int left = (int)c == pad_cl ? n - 8 * (int)c - 2 * t : 8;
                const char* x0 = x - (unsigned long long)(2 * t) * x_row;
                p0 = left > 0 ? p0 : x0;
                p1 = left > 1 ? p1 : x0;
            }
            v[2 * i] = __ldg(reinterpret_cast<const V*>(p0));
            v[2 * i + 1] = __ldg(reinterpret_cast<const V*>(p1));
        }
        tk[0] = tk[1] = 0u;
    } else {
        const unsigned* toks = reinterpret_cast<const unsigned*>(tok) + t;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            tk[i] = toks[(u + i) * 4];
            const unsigned a = tk[i] & 0xffffu, b = tk[i] >> 16;
            if (PICK::kHoles) {
                zero4(v[2 * i]);
                zero4(v[2 * i + 1]);
            }
            if (!PICK::kHoles || a != kSkip) v[2 * i] = __ldg(reinterpret_cast<const V*>(x + (unsigned long long)a * x_row));
            if (!PICK::kHoles || b != kSkip) v[2 * i + 1] = __ldg(reinterpret_cast<const V*>(x + (unsigned long long)b * x_row));
        }
    }
}
// Row of slot g of group u (nullptr: absent).  x: the head's rows (RUNS: at row g)
template <typename PICK>
__device__ __forceinline__ const char* slot_ptr(const char* x, unsigned x_row, const GroupSmem& sm, const unsigned short* tok, int u, int g,
                                                int pad_cl, int n) {
    if constexpr (PICK::kRuns) {
        const unsigned c = sm.rec.cl[u];
        const char* p = x + (unsigned long long)(8u * c) * x_row;
        if (PICK::kTail) p = (int)c == pad_cl && 8 * (int)c + g >= n ? x - (unsigned long long)g * x_row : p;
        return p;
    } else {
        const unsigned row = tok[u * 8 + g];
        if (PICK::kHoles && row == kSkip) return nullptr;
        return x + (unsigned long long)row * x_row;
    }
}
// ---- neighbour rows as the A operand (channels x slots) of out^T = X^T * W^T, for kernels with registers and issue slots to spare
// A request costs the L1 one cycle per (quarter of the warp, 128-byte line) for 16-byte loads -- per (half, line) for 8-byte
// ones -- so the layout that the operand wants, 4 slots by t, would cost 16 cycles for 512 bytes.  Rows are loaded as the L1
// likes them and moved to their lanes by instructions of one cycle each:
//   fp32    lane L reads 16 bytes, channels 4 (L % 8) .., of the slot of L / 8: 4 cycles, and 4 shuffles bring lane (g, t)
//           channels 4g .. 4g+3 of the slot of t
//   16-bit  lane (g, t) reads channels 8t .. 8t+7 of slot g: 8 cycles (4 when neighbouring tokens share a line), and 4
//           transpositions (movmatrix) give register r of slots 2t, 2t + 1 for channel 8 (g / 2) + 2r + g % 2
__device__ __forceinline__ float4 to_slots(const float4& v, int lane) {
    const int from = 8 * (lane & 3) + (lane >> 2);
    return make_float4(__shfl_sync(kFull, v.x, from), __shfl_sync(kFull, v.y, from), __shfl_sync(kFull, v.z, from), __shfl_sync(kFull, v.w, from));
}
__device__ __forceinline__ unsigned transpose8(unsigned v) {
    unsigned r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
    return r;
}
// 16-bit: M tiles 0, 1 from 8 + 8 slots
__device__ __forceinline__ void frag_slots16(unsigned (&a)[2][4], const uint4& x, const uint4& y) {
    a[0][0] = transpose8(x.x);  a[0][1] = transpose8(x.y);  a[1][0] = transpose8(x.z);  a[1][1] = transpose8(x.w);
    a[0][2] = transpose8(y.x);  a[0][3] = transpose8(y.y);  a[1][2] = transpose8(y.z);  a[1][3] = transpose8(y.w);
}
// 16-bit: a lane holds channels 8 (g / 2) + g % 2 + {0, 2, 4, 6} of both rows; lanes g, g ^ 1 swap one row each: v = channels
// 8 (g / 2) .. + 7 of row 2t + g % 2
__device__ __forceinline__ void acc_rows16(const float (&d)[2][4], int lane, float (&v)[8]) {
    const bool odd = (lane & 4) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float r0 = d[i >> 1][2 * (i & 1)], r1 = d[i >> 1][2 * (i & 1) + 1];
        const float got = __shfl_xor_sync(kFull, odd ? r0 : r1, 4);
        v[2 * i] = odd ? got : r0;
        v[2 * i + 1] = odd ? r1 : got;
    }
}

// The rows of groups u, u + 1 (u even), on their way to the A operand
template <typename T> struct RowRegs { uint4 v[2]; };
template <> struct RowRegs<float> { float4 v[4]; };
// x: the head's rows, at channel 8t (16-bit) or 4 (lane % 8) (fp32);  RUNS: at row g (16-bit) or 2 (lane / 8) (fp32)
template <typename PICK, typename T>
__device__ __forceinline__ void load_rows(RowRegs<T>& r, const char* x, unsigned x_row, const GroupSmem& sm, const unsigned short* tok, int u, int lane,
                                          int pad_cl, int n) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const char* p = slot_ptr<PICK>(x, x_row, sm, tok, u + i, lane >> 2, pad_cl, n);
        if (PICK::kHoles) r.v[i] = make_uint4(0u, 0u, 0u, 0u);
        if (!PICK::kHoles || p) r.v[i] = __ldg(reinterpret_cast<const uint4*>(p));
    }
}
template <typename PICK>
__device__ __forceinline__ void load_rows(RowRegs<float>& r, const char* x, unsigned x_row, const GroupSmem& sm, const unsigned short* tok, int u, int lane,
                                          int pad_cl, int n) {
    const int q = lane >> 3;
    if constexpr (PICK::kRuns) {
        const unsigned cc = *reinterpret_cast<const unsigned*>(sm.rec.cl + u);
        const char* x1 = x + x_row;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned c = i == 0 ? cc & 0xffffu : cc >> 16;
            const char* p0 = x + (unsigned long long)(8u * c) * x_row;
            const char* p1 = x1 + (unsigned long long)(8u * c) * x_row;
            if (PICK::kTail) {                               // slots behind the last token: token 0
                const int left = (int)c == pad_cl ? n - 8 * (int)c - 2 * q : 8;
                const char* x0 = x - (unsigned long long)(2 * q) * x_row;
                p0 = left > 0 ? p0 : x0;
                p1 = left > 1 ? p1 : x0;
            }
            r.v[2 * i] = __ldg(reinterpret_cast<const float4*>(p0));
            r.v[2 * i + 1] = __ldg(reinterpret_cast<const float4*>(p1));
        }
    } else {
        const unsigned* toks = reinterpret_cast<const unsigned*>(tok) + q;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned tk = toks[(u + i) * 4], a = tk & 0xffffu, b = tk >> 16;
            if (PICK::kHoles) r.v[2 * i] = r.v[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!PICK::kHoles || a != kSkip) r.v[2 * i] = __ldg(reinterpret_cast<const float4*>(x + (unsigned long long)a * x_row));
            if (!PICK::kHoles || b != kSkip) r.v[2 * i + 1] = __ldg(reinterpret_cast<const float4*>(x + (unsigned long long)b * x_row));
        }
    }
}
// element offset of a lane's pointer inside a row, and its row inside a cluster
template <typename T> __device__ __forceinline__ int rows_channel(int lane) { return std::is_same<T, float>::value ? 4 * (lane & 7) : 8 * (lane & 3); }
template <typename T> __device__ __forceinline__ int rows_first(int lane) { return std::is_same<T, float>::value ? 2 * (lane >> 3) : lane >> 2; }

// Two groups' products: acc[e] += X^T * W^T for E sets of 8 rows;  b(e, i) -> the set's B registers of group u + i, as
// float2 (fp32) or a 16-bit pair
template <typename T, int E, typename BF>
__device__ __forceinline__ void rows_product(float (&acc)[E][2][4], const RowRegs<T>& r, int lane, BF&& bf) {
    if constexpr (std::is_same<T, float>::value) {
        // (added up by themselves first: see step_rows in scatter_groups.cu)
        float d[E][2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 x0 = to_slots(r.v[2 * i], lane), x1 = to_slots(r.v[2 * i + 1], lane);
            const float a[2][4] = {{x0.x, x0.y, x1.x, x1.y}, {x0.z, x0.w, x1.z, x1.w}};
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const float2 w = bf(e, i);
                const float b[2] = {w.x, w.y};
                if (i == 0) mma_pair_first(d[e], a, b);
                else mma_pair<true>(d[e], a, b);
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[e][0][i] += d[e][0][i];
                acc[e][1][i] += d[e][1][i];
            }
    } else {
        unsigned a[2][4];
        frag_slots16(a, r.v[0], r.v[1]);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const unsigned b[2] = {bf(e, 0), bf(e, 1)};
            mma16(acc[e][0], a[0], b, static_cast<const T*>(nullptr));
            mma16(acc[e][1], a[1], b, static_cast<const T*>(nullptr));
        }
    }
}
// channel of accumulator element 2 i + j of M tile mt (row 2t + j)
template <typename T> __device__ __forceinline__ int acc_channel(int g, int mt, int i) {
    return std::is_same<T, float>::value ? 4 * g + 2 * mt + i : 8 * (g >> 1) + (g & 1) + 4 * mt + 2 * i;
}
// The set's 8 output rows (those below `rows`) -> out (contiguous rows of 32)
__device__ __forceinline__ void store_set(const float (&d)[2][4], float* out, int rows, int lane) {
    const int g = lane >> 2, t = lane & 3;
    float* o = out + 2 * t * kC + 4 * g;
    if (2 * t < rows) st4(o, acc_channels(d, 0));
    if (2 * t + 1 < rows) st4(o + kC, acc_channels(d, 1));
}
// 16-bit, row stride c
template <typename T> __device__ __forceinline__ void store_rows8(const float (&d)[2][4], T* out, int c, int rows, int lane) {
    float v[8];
    acc_rows16(d, lane, v);
    const int row = 2 * (lane & 3) + ((lane >> 2) & 1);
    if (row < rows)
        *reinterpret_cast<uint4*>(out + (long long)row * c + 8 * (lane >> 3)) =
            make_uint4(pack2(v[0], v[1], static_cast<const T*>(nullptr)), pack2(v[2], v[3], static_cast<const T*>(nullptr)),
                       pack2(v[4], v[5], static_cast<const T*>(nullptr)), pack2(v[6], v[7], static_cast<const T*>(nullptr)));
}
__device__ __forceinline__ unsigned byte_of(unsigned w, int i) { return __byte_perm(w, 0u, 0x4440u + i); }

// ---- copies to shared memory and operands from there (16-bit); addresses are 32-bit shared ones
__device__ __forceinline__ void cp_async16_or_zero(unsigned dst, const void* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldmatrix_x2_trans(unsigned (&r)[2], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void stmatrix_x4(unsigned a, unsigned r0, unsigned r1, unsigned r2, unsigned r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(unsigned a, unsigned r0, unsigned r1, unsigned r2, unsigned r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ unsigned lds16(unsigned a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ unsigned lds32(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 lds128(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cp_async16_cg(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
// Rows of 64 bytes in shared memory: the 16-byte piece c of row r lies at place c ^ (r / 2) % 4, so that neither 8 rows' pieces c (ldmatrix)
// nor the four pieces of two rows (16-byte accesses) share a bank
__device__ __forceinline__ unsigned row_piece(int r, int c) { return 64u * r + 16u * (c ^ ((r >> 1) & 3)); }
// out^T accumulators (M tile mt: channels 16 mt + g, + 8; columns 2t, 2t + 1: rows) of 8 rows -> rows of 64 bytes at buf
template <typename T> __device__ __forceinline__ void acc_to_rows(const float (&d)[2][4], unsigned buf, int lane) {
    const T* e = nullptr;
    stmatrix_x4_trans(buf + row_piece(lane & 7, lane >> 3), pack2(d[0][0], d[0][1], e), pack2(d[0][2], d[0][3], e), pack2(d[1][0], d[1][1], e), pack2(d[1][2], d[1][3], e));
}

// Heads per warp.  A warp that serves all heads reads its tile's record once; when the tiles alone leave the chip short
// of warps (`warps` per SM), the heads are spread over several warps.
inline void split_heads(long long tiles, int heads, int* parts, int* per_part, int warps = 24) {
    const long long want = (long long)sm_count() * warps;
    int per = heads;
    while (per > 1 && tiles * ((heads + per - 1) / per) < want) per = (per + 1) / 2;
    *per_part = per;
    *parts = (heads + per - 1) / per;
}

}  // namespace
}  // namespace clusten
