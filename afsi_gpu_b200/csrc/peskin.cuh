// Peskin IB_4 one-dimensional weights shared by the prepare kernels.
#pragma once
#include "common.cuh"

namespace afsi {

// Clamped two-branch Peskin kernel, afsi_torch/ib.py:57-67.  Only the branch
// that applies is evaluated (one square root): the taps of one offset fall in
// the same branch for all points but those on a grid line.
template <class T>
__device__ __forceinline__ T peskin_clamped(T d) {
    const T r = fabs(d);
    if (r < T(1)) return (T(3) - T(2) * r + sqrt(T(1) + T(4) * r - T(4) * (r * r))) / T(8);
    if (r < T(2)) return (T(5) - T(2) * r - sqrt(T(-7) + T(12) * r - T(4) * (r * r))) / T(8);
    return T(0);
}

// Shared-radical weights for f in [0,1), mac/csrc/p2_transfer.cu:36-43.
template <class T>
__device__ __forceinline__ void peskin_radical(T f, T w[4]) {
    const T rad = sqrt(T(1) + T(4) * f - T(4) * (f * f));
    w[0] = (T(3) - T(2) * f - rad) / T(8);
    w[1] = (T(3) - T(2) * f + rad) / T(8);
    w[2] = (T(1) + T(2) * f + rad) / T(8);
    w[3] = (T(1) + T(2) * f - rad) / T(8);
}

}  // namespace afsi
