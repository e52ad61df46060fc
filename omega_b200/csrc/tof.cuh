// TOF weights of the ray-driven projectors (types 1 and 4) over a sliding
// window of bins.
//
// A ray advances monotonically through the TOF bins, and a bin's Gaussian is
// nothing next to the element's total once its centre is much farther away than
// the nearest one's.  So a thread keeps W neighbouring bins in registers, in the
// order the ray meets them, instead of all of them: when the next bin outside
// the window comes nearer than the first one inside, the first is written out
// (forward) or dropped (backward) and the window moves on.  The host picks the
// smallest built W that leaves out only bins 8 sigma away whose weight is below
// 2^-30 of the element's total (tof_setup); with closely spaced bins that is
// every bin and nothing slides.  (An infinity or NaN in a measurement or voxel
// reaches the bins of the window, not all.)
//
// The weight of a bin is the 4-point trapezoid of its Gaussian over the
// element (TOFLoop / TOFWeight, general_opencl_functions.h:1077-1117).  About
// the element's middle m (distance over sigma sqrt 2, points b = element / 3
// apart in the same unit) the four exponentials share one:
//   e(m+1.5b) + e(m-1.5b) + 2 (e(m+b/2) + e(m-b/2))
//     = exp(-m^2) C [exp(-9 b^2/4) (C^2 - 3) + 2 exp(-b^2/4)],  C = 2 cosh(m b),
// and C is a short even series of m b: one special-function operation per bin
// instead of four, which is what bound these kernels (60 of them per sample
// of 15 bins, at 16 a clock and SM).  The series is used while b <= 0.3 (its
// remainder is below 2e-8 of it out to m = 4, where the weight is 1e-7), its argument
// clamped far from the bin (without the clamp a bin beyond m b = 81, 1.2 m for sigma 3 mm
// and elements of 3.5 mm, weighed 0 times infinity; the clamp costs 1 to 2 per cent); wider
// elements take the four exponentials.  Two bins go through each packed FP32 operation.
// Measured against every bin with four exponentials: 15 bins 4.5 sigma apart
// (W = 4), type 4, one 916,608-ray subset of 200 x 200 x 109 forward and back,
// 8.44 -> 3.46 ms; 9 bins about 1.9 sigma apart (every bin in the window),
// type 1, 1.09 -> 0.77 ms.  Error against 64 bits unchanged (4.3e-7).
#pragma once
#include "common.cuh"

namespace omb {

__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The built window sizes: even, so that bins pair up.
#define OMB_TOF_WINDOWS(X) X(2) X(4) X(6) X(8) X(10) X(12) X(14) X(16)

// Two FP32 values in one 64-bit register (Blackwell's packed FP32 pipe).
struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 x, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 both(float a) { return pack2(a, a); }

// The W bins a ray currently meets.  Positions p are distances along the ray's
// direction of travel (p = dir * D grows from element to element); nc holds
// the negated bin centres in that direction, a the bins' sums (forward) or
// measurements (backward).
template <int W>
struct TofWindow {
    float nc[W], a[W];
    float dir, th;   // th: position where the window moves on by one bin
    float moving;    // 1, or 0 when the ray starts exactly at its middle (every element then lies there)
    int k;           // bins before the window

    // centre and output slot of the k-th bin met
    __device__ __forceinline__ float centre(const Tof &t, int j) const {
        return dir * __ldg(t.sorted + (dir > 0.f ? j : t.nbins - 1 - j));
    }
    __device__ __forceinline__ int slot(const Tof &t, int j) const {
        const int i = dir > 0.f ? j : t.nbins - 1 - j;
        return t.order ? __ldg(t.order + i) : i;
    }
    __device__ __forceinline__ void threshold(const Tof &t) {
        th = k + W < t.nbins ? 0.5f * (centre(t, k) + centre(t, k + W)) : 3.4e38f;
    }
    __device__ __forceinline__ void begin(const Tof &t, float ddsign) {
        dir = ddsign > 0.f ? -1.f : 1.f;
        moving = fabsf(ddsign);
        k = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            nc[i] = i < t.nbins ? -centre(t, i) : 0.f;
            a[i] = 0.f;
        }
        threshold(t);
    }
    // moves on by one bin, whose sum / measurement becomes v
    __device__ __forceinline__ void advance(const Tof &t, float v) {
#pragma unroll
        for (int i = 0; i + 1 < W; ++i) {
            nc[i] = nc[i + 1];
            a[i] = a[i + 1];
        }
        nc[W - 1] = -centre(t, k + W);
        a[W - 1] = v;
        ++k;
        threshold(t);
    }

    // Weights of the window's bins for an element of length `ele` whose middle
    // lies at p, and their sum.  Returns what a weight is multiplied with:
    // scale / max(sum of the element's weights, epps).
    __device__ __forceinline__ float weights(const Tof &t, float p, float ele, float *w, float &sum) const {
        const float scale = t.sigma_coef * (ele / 3.f);
        const float eb = ele * moving;
        if (t.series) {
            const float e2 = eb * eb;
            const float x1 = ex2_approx(-e2 * t.kq);
            const float x3 = x1 * x1 * x1;
            const f32x2 q9 = both(x3 * x3 * x3), q1 = both(2.f * x1), kv = both(e2 * t.kv), k2 = both(-t.k2), p2 = both(p);
            f32x2 s2 = both(0.f);
#pragma unroll
            for (int i = 0; i < W; i += 2) {
                const f32x2 m = add2(p2, pack2(nc[i], nc[i + 1]));
                const f32x2 q = mul2(m, m);
                float x0, y0;
                unpack2(mul2(q, k2), x0, y0);
                // with an odd number of bins and all of them in the window, its last entry is no bin
                const f32x2 E = pack2(ex2_approx(x0), i + 2 == W && t.nbins < W ? 0.f : ex2_approx(y0));
                // far from the bin E is 0 and the series need only stay finite: C c^2 overflows from v = 6600, and
                // where E is not 0 v is below 8
                float v0, v1;
                unpack2(mul2(q, kv), v0, v1);
                const f32x2 v = pack2(fminf(v0, 100.f), fminf(v1, 100.f));
                f32x2 c = fma2(v, both(1.f / 1814400.f), both(1.f / 20160.f));
                c = fma2(v, c, both(1.f / 360.f));
                c = fma2(v, c, both(1.f / 12.f));
                c = fma2(v, c, both(1.f));
                c = fma2(v, c, both(2.f));
                const f32x2 g = fma2(q9, fma2(c, c, both(-3.f)), q1);
                const f32x2 ww = mul2(mul2(E, c), g);
                s2 = add2(s2, ww);
                unpack2(ww, w[i], w[i + 1]);
            }
            float sa, sb;
            unpack2(s2, sa, sb);
            sum = sa + sb;
        } else {
            const float si = t.sigma_inv * 0.70710678f;
            const float b = eb * (1.f / 3.f) * si;
            sum = 0.f;
#pragma unroll
            for (int i = 0; i < W; ++i) {
                const float m = (p + nc[i]) * si;
                const float a0 = fmaf(1.5f, b, m), a1 = fmaf(.5f, b, m), a2 = fmaf(-.5f, b, m), a3 = fmaf(-1.5f, b, m);
                w[i] = (__expf(-(a0 * a0)) + __expf(-(a3 * a3))) + 2.f * (__expf(-(a1 * a1)) + __expf(-(a2 * a2)));
                if (i + 1 == W && t.nbins < W) w[i] = 0.f;
                sum += w[i];
            }
        }
        return scale / fmaxf(sum * scale, t.epps);
    }
};

// The window rule (host).  `centers` (n of them) on the host; `element` the
// longest element a ray can have.  Fills sorted / order (n entries each) and
// t's window fields; without `sorted` every bin stays in the window.
inline void tof_setup(Tof &t, const float *centers, float *sorted, int *order, float element) {
    const int n = t.nbins;
    const double sigma = 1.0 / (double)t.sigma_inv, log2e = 1.4426950408889634;
    t.k2 = (float)(log2e / (2.0 * sigma * sigma));
    t.kv = (float)(1.0 / (36.0 * sigma * sigma * sigma * sigma));
    t.kq = (float)(log2e / (72.0 * sigma * sigma));
    const double b = element / 3.0 / (sigma * 1.4142135623730951);
    t.series = b <= 0.3;
    t.window = (n + 1) / 2 * 2;
    if (!sorted) return;
    bool finite = true;
    for (int i = 0; i < n; ++i) {
        order[i] = i;
        finite = finite && centers[i] - centers[i] == 0.f;
    }
    if (finite)
        for (int i = 1; i < n; ++i)   // insertion sort, n <= 16
            for (int j = i; j > 0 && centers[order[j]] < centers[order[j - 1]]; --j) {
                const int o = order[j];
                order[j] = order[j - 1];
                order[j - 1] = o;
            }
    for (int i = 0; i < n; ++i) sorted[i] = centers[order[i]];
    if (!finite) return;
    // The window moves on halfway between bins i and i + w.  There the bin left
    // out (or not yet met) weighs most against the element's total: farther on it
    // loses more than the nearest bin does.  The total is at least a third (the
    // trapezoid's inner points) of the nearest bin's Gaussian a sixth of an
    // element farther away.  Evenly spaced bins have one halfway and pass the
    // second test with the first; bins in pairs far apart need not.
    for (int w = 2; w < n; w += 2) {
        bool covers = true;
        for (int i = 0; i + w < n; ++i) {
            const double at = 0.5 * ((double)sorted[i] + sorted[i + w]), half = at - sorted[i];
            double nearest = half;
            for (int j = i + 1; j < i + w; ++j) nearest = fmin(nearest, fabs(at - sorted[j]));
            const double away = half - 0.5 * element, near = nearest + element / 6.0;
            // 3 exp(-x / 2 sigma^2) < 2^-30 from x = 43.8 sigma^2
            covers = covers && away >= 8.0 * sigma && away * away - near * near >= 44.0 * sigma * sigma;
        }
        if (covers) {
            t.window = w;
            return;
        }
    }
}

}  // namespace omb
