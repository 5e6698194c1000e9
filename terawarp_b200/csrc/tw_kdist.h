// tw_kdist.h -- the TPS kernel of two landmarks, shared by the solve's kernels
// (one definition, so that every kernel rounds it the same way).
#pragma once

namespace tw {

// K_ij = -|s_i - s_j|
__device__ __forceinline__ double kdist(const double *ctr, int i, int j)
{
    double dx = ctr[3 * i] - ctr[3 * j];
    double dy = ctr[3 * i + 1] - ctr[3 * j + 1];
    double dz = ctr[3 * i + 2] - ctr[3 * j + 2];
    return -sqrt(dx * dx + dy * dy + dz * dz);
}

}  // namespace tw
