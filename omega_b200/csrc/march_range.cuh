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

// Samples [lo, hi] of a march of n samples that lie inside on one axis (c + i s
// in [0, size - 1), with a margin far above the rounding of c + i s);
// intersected into lo, hi.  An axis of one voxel has no such sample: every one
// of its samples lies beside the voxel's centre, where the neighbour is the
// edge voxel itself.
OMB_MARCH_FN void inside_range(float c, float s, unsigned n, int size, float &lo, float &hi) {
    const float a = 0.01f - c, b = (float)(size - 1) - 0.01f - c;
    if (!(a <= b)) {
        hi = -1.f;
        return;
    }
    if (fabsf(s) < 1e-6f) {
        // nearly constant: inside from the first sample to the last (a march may
        // have 4e9 of them), or not at all
        const float e = (float)(n - 1) * s;
        if (!(fminf(0.f, e) >= a && fmaxf(0.f, e) <= b)) hi = -1.f;
        return;
    }
    const float p = a / s, q = b / s;
    lo = fmaxf(lo, ceilf(fminf(p, q)));
    hi = fminf(hi, floorf(fmaxf(p, q)));
}

// The range as sample counts: [0, first) and [last, n) need the clamps.  (A
// count above 2^24 may round up on its way to float and back.)
OMB_MARCH_FN void interior(float lo, float hi, unsigned n, unsigned &first, unsigned &last) {
    first = last = n;
    if (!(lo <= hi)) return;
    if (lo < 4e9f && (unsigned)lo < n) first = (unsigned)lo;
    if (hi < 4e9f && (unsigned)hi < n) last = (unsigned)hi + 1u;
}

}  // namespace omb
