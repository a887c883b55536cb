// Records of a neighbour table's tiles (group_core.cuh), one warp per tile of 16 rows.
//
// The backward passes of QK and AV in all blocks of a stage, and forward calls for which that pays by itself, then read 512 bytes
// per tile instead of 6 KB of int64 indices.  Bound by the one pass over the indices.
#include "group_core.cuh"

namespace clusten {
namespace {

constexpr int kPlanWarps = 8;

// ANY: rows that are no multiple of 8 long or do not start on 16-byte boundaries.  They have no whole clusters; a kernel without the code for those has
// registers to spare for divisions by multiplication: 256 tables of 49 rows of 49 8.3 -> 6.2 us.  (With `wide` known to be true as well the compiler
// takes 93 registers instead of 79.)
template <int RT, bool TAIL, bool ANY>
__global__ void __launch_bounds__(32 * kPlanWarps)
group_plan_kernel(const int64_t* __restrict__ idx, int n_rows, int m, int n_src, int wide, int tiles, unsigned total,
                  TileRecord* __restrict__ plan, uint2* __restrict__ columns) {
    __shared__ TileRecord recs[kPlanWarps];
    __shared__ __align__(16) unsigned char tags[kPlanWarps][kTagSpan];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned task = blockIdx.x * kPlanWarps + warp;
    if (task >= total) return;
    const unsigned b = task / (unsigned)tiles;
    const int i0 = (int)(task - b * (unsigned)tiles) * kTR;
    TileRecord& rec = recs[warp];
    build_record<RT, TAIL, !ANY>(idx + ((long long)b * n_rows + i0) * m, min(kTR, n_rows - i0), m, (m + 7) >> 3, n_src, !ANY && wide != 0, rec, tags[warp], lane);
    reinterpret_cast<uint4*>(plan + task)[lane] = reinterpret_cast<const uint4*>(&rec)[lane];
    // the map by group: 16 places of 4 bits, for the inverse (group_inverse.cu)
    if ((rec.head & 0xffu) == kRecRuns && lane < kMaxU) {
        unsigned lo = 0u, hi = 0u;
#pragma unroll
        for (int row = 0; row < 8; ++row) {
            lo |= (unsigned)rec.map[row][lane] << (4 * row);
            hi |= (unsigned)rec.map[row + 8][lane] << (4 * row);
        }
        columns[(size_t)task * kMaxU + lane] = make_uint2(lo, hi);
    }
}

}  // namespace

size_t group_plan_bytes(int b, int n_rows) { return (size_t)b * group_tiles(n_rows) * (sizeof(TileRecord) + kMaxU * sizeof(uint2)); }

bool group_plan_supported(int n_src, int m) { return m >= 1 && m <= kGroupMaxM && n_src >= 1 && n_src <= 65000; }

int launch_group_plan(const int64_t* idx, int b, int n_rows, int m, int n_src, void* plan, cudaStream_t s) {
    const int tiles = group_tiles(n_rows);
    if ((long long)b * tiles > 0x7fffffffLL) return CLUSTEN_ERR_SHAPE;
    const unsigned total = (unsigned)b * (unsigned)tiles;
    const bool wide = m % 8 == 0 && reinterpret_cast<uintptr_t>(idx) % 16 == 0;
    const bool tail = n_src % 8 != 0;
    auto kernel = !wide ? group_plan_kernel<0, true, true>
                        : (m == kMmax ? (tail ? group_plan_kernel<6, true, false> : group_plan_kernel<6, false, false>)
                                      : (tail ? group_plan_kernel<0, true, false> : group_plan_kernel<0, false, false>));
    ScopedKernelTimer timer("group_plan", s);
    kernel<<<(total + kPlanWarps - 1) / kPlanWarps, 32 * kPlanWarps, 0, s>>>(idx, n_rows, m, n_src, wide, tiles, total, static_cast<TileRecord*>(plan),
                                                                                   reinterpret_cast<uint2*>(static_cast<TileRecord*>(plan) + total));
    note_launch();
    return check_launch();
}

}  // namespace clusten
