// Inverse of a neighbour table by groups, from its records (group_core.cuh).
//
// The scatter-side gradients (scatter_groups.cu) give a warp the 8 targets 8T .. 8T+7.  What names them is stored per T, ordered
// by source row, so that the summation order is fixed:
//
//   kBuildGroupRuns    every record of the batch element is of kind "runs".  One 4-byte entry per row that names cluster T:
//                      row << 8 | place: slots 8 (place - 1) .. 8 (place - 1) + 7 are the targets.  A list is filled up to a
//                      multiple of 16 entries with zeros (place 0: nothing).
//   kBuildGroupLists   every record is of kind "same".  An entry of 16 bytes is 8 rows with one list that names one of the
//                      targets at least: {first row, 8 bytes}: the slot that is target 8T + q, 0xff: none.
//
// The buffer is the ordinary inverse index (common.cuh), with these entries where the per-target ones would be; rowptr and
// seglen hold their start and number per T.
// Batch elements that are neither get the ordinary index from inverse.cu.
// One CTA per batch element; which (rows, T) pairs exist is a bit mask in shared memory, set with integer ORs and read
// with population counts, so the result does not depend on the order of the atomics.
#include "group_core.cuh"

namespace clusten {
namespace {

constexpr int kGIThreads = 1024;
constexpr int kGIWarps = kGIThreads / 32;

// a bit for every digit of 4 bits that is not zero
__device__ __forceinline__ unsigned any_bit(unsigned v) { return (v | v >> 1 | v >> 2 | v >> 3) & 0x11111111u; }

__global__ void __launch_bounds__(kGIThreads)
group_inverse_kernel(const TileRecord* __restrict__ plan, int n_rows, int m, int nt, int ntiles, int words_cap, int* __restrict__ header,
                     int* __restrict__ rowptr, int* __restrict__ seglen, int* __restrict__ entries, int* __restrict__ tileflag) {
    extern __shared__ __align__(16) unsigned gi_sm[];
    unsigned* mask = gi_sm;                                    // [ntiles][words]
    int* base = reinterpret_cast<int*>(gi_sm + (size_t)ntiles * words_cap);      // [ntiles] first (rows, T) pair of target tile T
    int* cnt = base + ntiles;                                  // runs: [ntiles] rows that name T
    __shared__ int warp_tot[kGIWarps];
    __shared__ int total_s, total_l, again;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles = (n_rows + kTR - 1) / kTR;
    const TileRecord* recs = plan + (long long)b * tiles;
    const uint2* cols = reinterpret_cast<const uint2*>(plan + (long long)gridDim.x * tiles) + (long long)b * tiles * kMaxU;
    int* tf = tileflag + (long long)b * (1 + ntiles);
    if (b == 0 && tid < kInvHeaderInts)
        header[tid] = tid == 0 ? (int)kInvMagic : tid == 1 ? (int)gridDim.x : tid == 2 ? n_rows : tid == 3 ? m : tid == 4 ? nt : 0;
    bool runs = words_cap > 0, lists = words_cap > 0;
    if (words_cap > 0)
        for (int i = tid; i < tiles; i += kGIThreads) {
            const unsigned head = recs[i].head;
            runs = runs && (head & 0xffu) == kRecRuns;
            lists = lists && (head & 0x100ffu) == kRecSame;           // and no slot absent
        }
    runs = __syncthreads_and(runs);
    lists = __syncthreads_and(lists);
    if (!runs && !lists) {
        if (tid == 0) tf[0] = kBuildGeneral;
        return;
    }
    const int nlists = (n_rows + 7) >> 3;
    const int words = ((runs ? tiles : nlists) + 31) >> 5;
    for (int i = tid; i < ntiles * words; i += kGIThreads) mask[i] = 0u;
    for (int i = tid; i < ntiles; i += kGIThreads) cnt[i] = 0;
    if (tid == 0) again = 0;
    __syncthreads();
    // ---- which rows name which target tile
    for (int i = warp; i < tiles; i += kGIWarps) {
        if (runs) {
            const int U = (recs[i].head >> 8) & 0xff;
            if (lane < U) {
                const int T = recs[i].cl[lane];
                atomicOr(&mask[T * words + (i >> 5)], 1u << (i & 31));
                const uint2 c = __ldg(cols + i * kMaxU + lane);
                atomicAdd(&cnt[T], __popc(any_bit(c.x)) + __popc(any_bit(c.y)));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int l = 2 * i + e;
                if (l < nlists)
                    for (int j = lane; j < m; j += 32) atomicOr(&mask[(int)(recs[i].lists[e][j] >> 3) * words + (l >> 5)], 1u << (l & 31));
            }
        }
    }
    __syncthreads();
    // ---- pairs and list entries per target tile, and where they start
    {
        const int per = (ntiles + kGIThreads - 1) / kGIThreads;
        const int lo = min(tid * per, ntiles), hi = min(lo + per, ntiles);
        int local = 0, local_l = 0;
        for (int T = lo; T < hi; ++T) {
            int c = 0;
            for (int w = 0; w < words; ++w) c += __popc(mask[T * words + w]);
            base[T] = c;
            local += c;
            local_l += (cnt[T] + 15) >> 4;
        }
        // (both sums travel in one word: pair_counts_fit)
        unsigned incl = (unsigned)local | (unsigned)local_l << 16;
        const unsigned mine = incl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = (int)incl;
        __syncthreads();
        if (warp == 0) {
            const unsigned w = (unsigned)warp_tot[lane];
            unsigned wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(kFull, wi, o);
                if (lane >= o) wi += y;
            }
            warp_tot[lane] = (int)(wi - w);
            if (lane == 31) {
                total_s = (int)(wi & 0xffffu);
                total_l = (int)(wi >> 16);
            }
        }
        __syncthreads();
        const unsigned before = (unsigned)warp_tot[warp] + incl - mine;
        int run = (int)(before & 0xffffu), run_l = (int)(before >> 16);
        int* rp = rowptr + (long long)b * (nt + 1);
        int* sl = seglen + (long long)b * nt;
        for (int T = lo; T < hi; ++T) {
            const int c = base[T], steps = (cnt[T] + 15) >> 4;
            base[T] = run;
            rp[T] = runs ? 16 * run_l : run;
            sl[T] = runs ? 16 * steps : c;
            if (runs) {                                        // where group_lists_kernel finds the pairs
                rp[ntiles + T] = run;
                sl[ntiles + T] = c;
            }
            run += c;
            run_l += steps;
        }
    }
    // runs: the pairs are written behind where the lists go
    unsigned* list = reinterpret_cast<unsigned*>(group_entries(entries, b, n_rows, m));
    uint4* ent = reinterpret_cast<uint4*>(list) + (runs ? 4 * total_l : 0);
    if (lists)
        for (int i = tid; i < total_s; i += kGIThreads) ent[i] = make_uint4(0u, 0xffffffffu, 0xffffffffu, 0u);
    __syncthreads();
    if (runs && 4 * (total_s + 4 * total_l) + 4 > n_rows * m) {      // no room: such a table is left to the ordinary build
        if (tid == 0) tf[0] = kBuildGeneral;
        return;
    }
    auto place = [&](int T, int i) {                           // entry of source i (tile or list) of target tile T
        const unsigned* mk = mask + T * words;
        int pos = base[T] + __popc(mk[i >> 5] & ((1u << (i & 31)) - 1u));
        for (int w = 0; w < (i >> 5); ++w) pos += __popc(mk[w]);
        return pos;
    };
    if (runs) {
        // a pair: {first row, 16 places of 4 bits}, in the order of the rows
        for (int i = warp; i < tiles; i += kGIWarps) {
            const int U = (recs[i].head >> 8) & 0xff;
            if (lane < U) {
                const uint2 c = __ldg(cols + i * kMaxU + lane);
                ent[place((int)recs[i].cl[lane], i)] = make_uint4((unsigned)(i * kTR), c.x, c.y, 0u);
            }
        }
        if (tid == 0) {
            tf[0] = kBuildGroupRuns;
            rowptr[(long long)b * (nt + 1) + nt] = 4 * total_l;       // pairs start here (in 16 bytes)
        }
        return;
    }
    unsigned char* bytes = reinterpret_cast<unsigned char*>(ent);
    for (int l = warp; l < nlists; l += kGIWarps)
        for (int j = lane; j < m; j += 32) {
            const int tok = recs[l >> 1].lists[l & 1][j];
            const int pos = place(tok >> 3, l);
            ent[pos].x = (unsigned)(8 * l);
            bytes[16 * (long long)pos + 4 + (tok & 7)] = (unsigned char)j;
        }
    __syncthreads();
    // a list that names a token twice has overwritten its own slot: such a batch element is left to the ordinary build
    for (int l = warp; l < nlists; l += kGIWarps)
        for (int j = lane; j < m; j += 32) {
            const int tok = recs[l >> 1].lists[l & 1][j];
            if (bytes[16 * (long long)place(tok >> 3, l) + 4 + (tok & 7)] != j) again = 1;
        }
    __syncthreads();
    if (tid == 0) tf[0] = again ? kBuildGeneral : kBuildGroupLists;
}

// The lists of the target tiles, from the pairs that group_inverse_kernel left behind them: a warp per tile.
__global__ void __launch_bounds__(256)
group_lists_kernel(int n_rows, int m, int nt, int ntiles, unsigned total, const int* __restrict__ rowptr, const int* __restrict__ seglen,
                   const int* entries, const int* __restrict__ tileflag) {
    const int lane = threadIdx.x & 31;
    const unsigned task = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (task >= total) return;
    const int b = (int)(task / (unsigned)ntiles), T = (int)(task - (unsigned)b * (unsigned)ntiles);
    if (tileflag[(long long)b * (1 + ntiles)] != kBuildGroupRuns) return;
    const int* rp = rowptr + (long long)b * (nt + 1);
    const int* sl = seglen + (long long)b * nt;
    unsigned* list = reinterpret_cast<unsigned*>(group_entries(entries, b, n_rows, m));
    const uint4* ent = reinterpret_cast<const uint4*>(list) + rp[nt] + rp[ntiles + T];
    const int count = sl[ntiles + T], end = rp[T] + sl[T];
    int at = rp[T];
    const int row = lane & 15;
    for (int k0 = 0; k0 < count; k0 += 32) {
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
        if (k0 + lane < count) e = ent[k0 + lane];
        // two pairs at a time, a lane per row: what a trip writes is contiguous
        for (int k = 0; k < min(32, count - k0); k += 2) {
            const int from = k + (lane >> 4);
            const unsigned first = __shfl_sync(kFull, e.x, from), lo = __shfl_sync(kFull, e.y, from), hi = __shfl_sync(kFull, e.z, from);
            const unsigned v = ((row & 8 ? hi : lo) >> (4 * (row & 7))) & 15u;      // (pairs behind the last one are zero)
            const unsigned named = __ballot_sync(kFull, v != 0u);
            if (v) list[at + __popc(named & ((1u << lane) - 1u))] = (first + row) << 8 | v;
            at += __popc(named);
        }
    }
    if (at + lane < end) list[at + lane] = 0u;
}

}  // namespace

// Shared memory of group_inverse_kernel; 0: too many rows for the bit mask or the counters, or so few that the entries might not fit
// their place
static size_t group_inverse_smem(int n_rows, int m, int nt) {
    const int ntiles = inverse_tiles(nt), words = ((n_rows + 7) / 8 + 31) / 32;
    const size_t smem = ((size_t)ntiles * words + 2 * (size_t)ntiles) * sizeof(int);
    return smem > 200 * 1024 || n_rows < 16 || !pair_counts_fit(n_rows, m) ? 0 : smem;
}

bool group_inverse_applies(int n_rows, int m, int nt) { return group_plan_supported(nt, m) && group_inverse_smem(n_rows, m, nt) != 0; }

int launch_group_inverse(const int64_t* idx, const void* plan, int b, int n_rows, int m, int nt, void* buf, cudaStream_t s) {
    int* p = static_cast<int*>(buf);
    const InverseView v = inverse_view(buf, b, n_rows, m, nt);
    const int ntiles = inverse_tiles(nt);
    const size_t smem = group_inverse_smem(n_rows, m, nt);
    const int words = smem != 0 ? ((n_rows + 7) / 8 + 31) / 32 : 0;          // (0: the ordinary build does everything)
    const int fit = resident_ctas(reinterpret_cast<const void*>(group_inverse_kernel), kGIThreads, smem);
    if (fit < 0) return fit;
    {
        ScopedKernelTimer timer("inverse_build", s);
        group_inverse_kernel<<<b, kGIThreads, smem, s>>>(static_cast<const TileRecord*>(plan), n_rows, m, nt, ntiles, words, p, const_cast<int*>(v.rowptr),
                                                         const_cast<int*>(v.seglen), const_cast<int*>(v.entries), const_cast<int*>(v.tileflag));
        note_launch();
        int st = check_launch();
        if (st != CLUSTEN_OK) return st;
        if (words > 0 && m % 8 == 0) {                         // (other tables have no clusters)
            const unsigned total = (unsigned)b * (unsigned)ntiles;
            ScopedKernelTimer timer2("inverse_build", s);
            group_lists_kernel<<<(total + 7) / 8, 256, 0, s>>>(n_rows, m, nt, ntiles, total, v.rowptr, v.seglen, v.entries, v.tileflag);
            note_launch();
            st = check_launch();
            if (st != CLUSTEN_OK) return st;
        }
    }
    return launch_inverse_general(idx, b, n_rows, m, nt, buf, s);
}

}  // namespace clusten
