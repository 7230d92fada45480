// Ray-box test of the throughput traversal (wavefront.cu), in plain float arithmetic that
// also compiles for the host, where tests/cpp/slab.cpp compares it with the two-sided form.
#pragma once
#include <cmath>

#include "pt_layout.h"

namespace ptg {

// Three-input maximum and minimum (max.f32 / min.f32 with three sources, sm_100 and
// later); a NaN operand is ignored, as by fmaxf / fminf.
PT_HD float Max3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
PT_HD float Min3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
#else
    return fminf(fminf(a, b), c);
#endif
}

// Whether a ray meets an axis's upper planes first (1) or its lower ones (0): the sign of
// its direction component, from inv = 1 / d and oi = o / d. Choosing once per ray spares
// the slab tests a minimum and a maximum per axis and child; these run at half the rate of
// the multiply-adds, and the traversal is bound by issue. Where 1 / d or o / d overflows,
// a plane distance is infinite or NaN, and the choice is the other way round: then the
// interval is empty exactly where taking the smaller and the larger of an axis's two
// distances (a NaN ignored) leaves it empty, so both forms visit the same boxes (an
// infinite direction needs boxes that are finite, or infinite on both sides, as the tree's
// are).
//
// They are not all the boxes that such a ray meets. With a direction component of exactly zero,
// or so small that 1 / d or o / d overflows, and an origin other than zero there, a box whose
// planes on that axis lie on both sides of zero is left out even where it holds the origin
// between them: one plane's distance is infinite, the other NaN. Axis-parallel rays of a query
// avoid it (SlabInverse). Other rays with one such component do not, in queries and among an image's
// paths: about one in 3M random rays, a few of the 132.7M paths of a 1080p frame, which may miss a hit
// or an occluder. Their results are kept bit for bit as they have been.
PT_HD int UpperFirst(float inv, float oi) {
    const float most = 3.402823466e+38f;
    const bool over = fabsf(inv) > most || fabsf(oi) > most;
    return (copysignf(1.0f, inv) < 0.0f) != over ? 1 : 0;
}

// Whether 1 / d or o / d overflows.
PT_HD bool SlabOverflows(float inv, float o) {
    const float most = 3.402823466e+38f;
    return fabsf(inv) > most || fabsf(o * inv) > most;
}
// The reciprocal for the slab test of one axis of an axis-parallel ray: 1 / d, or +-2^64 where it
// or o / d overflows, a component of 2^-64 in the direction's place. A power of two times the origin
// is exact, so a plane's distance is (plane - o) 2^64 rounded once: negative before the origin,
// beyond any hit after it, and never NaN for coordinates below 2^64. So the plainest rays of
// picking and baking meet the boxes that they pass through. Once per ray of a query; in the wave's
// kernels it costs 1 to 2% of a frame.
constexpr float kSlabMost = 18446744073709551616.0f;  // 2^64
PT_HD float SlabInverse(float inv, float o) {
    return SlabOverflows(inv, o) ? copysignf(kSlabMost, inv) : inv;
}
// A ray is axis-parallel with two components below 2^-64, zero or not.
PT_HD bool AxisParallel(float ix, float iy, float iz) {
    return (fabsf(ix) > kSlabMost) + (fabsf(iy) > kSlabMost) + (fabsf(iz) > kSlabMost) >= 2;
}

// Entry distance of a box's overlap with [0, tmax], +infinity where there is none, from the
// three planes the ray meets first (n) and the three it meets last (f). Each plane
// distance is one fused multiply-add, plane * inv - oi. Its rounding (a few units in the
// last place of the origin's and the distance's coordinates) is far inside the 2^-18
// widening of the child boxes, so no hit box is missed while inv and oi are finite
// (UpperFirst says what happens otherwise).
PT_HD float SlabEntry(float nx, float ny, float nz, float fx, float fy, float fz, float ix, float iy,
                      float iz, float ox, float oy, float oz, float tmax) {
    const float tn = Max3(fmaf(nx, ix, -ox), fmaf(ny, iy, -oy), fmaxf(fmaf(nz, iz, -oz), 0.0f));
    const float tf = Min3(fmaf(fx, ix, -ox), fmaf(fy, iy, -oy), fminf(fmaf(fz, iz, -oz), tmax));
    return tn <= tf ? tn : INFINITY;
}

}  // namespace ptg
