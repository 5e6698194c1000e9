// tw_kdist.h -- the TPS kernel of two landmarks, shared by the solve's kernels
// (one definition, so that every kernel rounds it the same way).
#pragma once

namespace tw {

// -|a - b|
__device__ __forceinline__ double kdist(double ax, double ay, double az, double bx, double by, double bz)
{
    double dx = ax - bx;
    double dy = ay - by;
    double dz = az - bz;
    return -sqrt(dx * dx + dy * dy + dz * dz);
}

}  // namespace tw
