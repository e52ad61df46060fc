// Which samples of a type-4 march may be interpolated without clamps
// (trilinear_inside, interp.cu).  Plain C++ besides the qualifier, so that the
// test suite compiles it for the host and tries every sample of a range.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define OMB_MARCH_FN __device__ __forceinline__
#else
#define OMB_MARCH_FN inline
#endif

namespace omb {

// Samples [lo, hi] of a march that lie inside on one axis (c + n s in [0, size
// - 1), with a margin far above the rounding of c + n s); intersected into lo,
// hi.  An axis of one voxel has no such sample: every one of its samples lies
// beside the voxel's centre, where the neighbour is the edge voxel itself.
OMB_MARCH_FN void inside_range(float c, float s, int size, float &lo, float &hi) {
    const float a = 0.01f - c, b = (float)(size - 1) - 0.01f - c;
    if (!(a <= b)) {
        hi = -1.f;
        return;
    }
    if (fabsf(s) < 1e-6f) {
        // (a sample count times 1e-6 stays far inside one voxel)
        if (!(a <= -0.5f && b >= 0.5f)) hi = -1.f;
        return;
    }
    const float p = a / s, q = b / s;
    lo = fmaxf(lo, ceilf(fminf(p, q)));
    hi = fminf(hi, floorf(fmaxf(p, q)));
}

}  // namespace omb
