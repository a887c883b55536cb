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

}  // namespace clusten
