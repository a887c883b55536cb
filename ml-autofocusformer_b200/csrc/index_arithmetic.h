// Index arithmetic of the group kernels that a host compiler can read too.
#pragma once

#ifdef __CUDACC__
#define CLUSTEN_HD __host__ __device__ __forceinline__
#else
#define CLUSTEN_HD inline
#endif

namespace clusten {

// Places (0: not named) of the groups first .. first + 3 in a row that is a list of `groups` groups, a byte each.  Rows from
// `rows` on do not exist and name nothing: a consumer that looks a row's operand up by place (the dense biases of the fused
// attention, which lie behind one another) must not be sent there.
CLUSTEN_HD unsigned list_places(int row, int first, int groups, int rows) {
    unsigned b = 0u;
    for (int i = 0; i < 4; ++i) b |= (row < rows && first + i < groups ? (unsigned)(first + i + 1) : 0u) << (8 * i);
    return b;
}

// Do the (source, target tile) pairs of one batch element fit the 16 bits that group_inverse_kernel counts them in?  Sources are
// tiles of 16 rows with whole clusters (a row names at most ceil(m / 8) of them) or lists of 8 rows, of which every slot can
// name another target tile.
CLUSTEN_HD bool pair_counts_fit(int n_rows, int m) {
    return (long long)n_rows * ((m + 7) / 8) <= 65535 && (long long)((n_rows + 7) / 8) * m <= 65535;
}

}  // namespace clusten
