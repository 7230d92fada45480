// The slab test of a caller's ray (csrc/slab.h SlabInverse, UpperFirst, SlabEntry) against
// the exact overlap in 64 bits, for directions with one or two components that are zero (either
// sign) or too small for their reciprocal, over boxes on all sides of the origin: a box that
// holds the ray on those axes by its widening is hit at the entry distance of the other axes, and
// one that does not is missed. Prints "ok <cases>" or the first difference.
#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "slab.h"

int main() {
    const float none[] = {0.0f, -0.0f, 1.0e-45f, -1.0e-45f, 1.0e-39f, -2.0e-39f, 1.0e-37f};
    const float origins[] = {0.0f, -0.0f, 1.0f, -3.0f, 1.0e-6f, 250.0f, -1.0e7f};
    const float widths[] = {2.0e-3f, 1.0f, 300.0f};   // of the box around the origin, in units of max(1, |o|)
    const float sides[] = {-900.0f, -1.5f, -0.6f, 0.0f, 0.6f, 1.5f, 900.0f};  // box centre, in widths from the origin
    const float dirs[] = {1.0f, -1.0f, 0.25f, -3.0e-5f};
    long cases = 0, hits = 0;
    for (float d0 : none)
        for (float o0 : origins)
            for (float w : widths)
                for (float at : sides)
                    for (int two = 0; two < 2; two++)
                        for (float dz : dirs)
                            for (float z0 : {-7.0f, 0.5f, 6.0f})
                                for (float tmax : {3.402823466e+38f, 8.0f}) {
                                    const float size = w * fmaxf(1.0f, fabsf(o0)), c = o0 + at * size;
                                    const float lo[3] = {c - size / 2, -2.0f, z0}, hi[3] = {c + size / 2, 3.0f, z0 + 2.0f};
                                    const float o[3] = {o0, 1.0f, 0.25f}, d[3] = {d0, two ? d0 : 0.125f, dz};
                                    float inv[3], oi[3], n[3], f[3];
                                    double t0 = 0.0, t1 = tmax;
                                    bool in = true;
                                    for (int k = 0; k < 3; k++) {
                                        inv[k] = ptg::SlabInverse(1.0f / d[k], o[k]);
                                        oi[k] = o[k] * inv[k];
                                        const int up = ptg::UpperFirst(inv[k], oi[k]);
                                        n[k] = up ? hi[k] : lo[k];
                                        f[k] = up ? lo[k] : hi[k];
                                        if (fabsf(d[k]) < 1.0e-30f) {
                                            in = in && lo[k] < o[k] && o[k] < hi[k];
                                        } else {
                                            const double a = ((double)lo[k] - o[k]) / d[k], b = ((double)hi[k] - o[k]) / d[k];
                                            t0 = fmax(t0, fmin(a, b));
                                            t1 = fmin(t1, fmax(a, b));
                                        }
                                    }
                                    if (fabs(t1 - t0) < 1.0e-3 * fmax(1.0, fabs(t0))) continue;  // a touch either way
                                    const float got = ptg::SlabEntry(n[0], n[1], n[2], f[0], f[1], f[2], inv[0], inv[1],
                                                                     inv[2], oi[0], oi[1], oi[2], tmax);
                                    const bool want = in && t0 < t1;
                                    cases++;
                                    hits += want;
                                    if (want ? !(fabs(got - t0) <= 1.0e-4 * fmax(1.0, fabs(t0))) : !std::isinf(got))
                                        return std::printf("o %g d %g %g %g box %g..%g z %g tmax %g: got %g want %g\n", o0, d[0],
                                                           d[1], d[2], lo[0], hi[0], z0, tmax, got, want ? t0 : INFINITY), 1;
                                }
    // ordinary directions keep their reciprocal
    for (float d : {1.0f, -0.3f, 1.0e-20f, INFINITY, -INFINITY})
        if (ptg::SlabInverse(1.0f / d, 5.0f) != 1.0f / d) return std::printf("1 / %g changed\n", d), 1;
    const float inf = INFINITY;
    if (ptg::AxisParallel(inf, 2.0f, -1.0f) || ptg::AxisParallel(NAN, inf, 1.0f) || !ptg::AxisParallel(inf, 1.0f, -1.0e38f) ||
        !ptg::AxisParallel(-inf, inf, 1.0f) || !ptg::AxisParallel(0.0f, -1.0e20f, inf))
        return std::printf("axis-parallel rays mistaken\n"), 1;
    if (!std::isnan(ptg::SlabInverse(NAN, 1.0f))) return std::printf("NaN changed\n"), 1;
    std::printf("ok %ld %ld\n", cases, hits);
    return 0;
}
