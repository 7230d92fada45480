// SlabEntry with the planes chosen once per ray (UpperFirst, csrc/slab.h) against the
// two-sided form, which takes the smaller and the larger distance of every axis (a NaN
// ignored): the same box hit or missed and the same entry distance, for every combination
// of an axis's bounds, origin and direction over ordinary values, signed zeros, tiny and
// huge numbers, infinities and NaN. Two axes vary at a time (through the same axis table),
// the third is ordinary. Prints "ok <cases>" or the first difference.
#include <cmath>
#include <cstdio>
#include <vector>

#include "slab.h"

struct Axis {
    float lo, hi, o, d, inv, oi;
};

int main() {
    const float inf = INFINITY, nan = NAN;
    const float bounds[] = {-inf, -3.0e38f, -5.0f, -1.0e-3f, -1.0e-40f, -0.0f, 0.0f, 1.0e-40f, 1.0e-3f, 4.0f, 3.0e38f, inf};
    const float origins[] = {-3.0e38f, -6.0f, -4.0f, -1.0e-39f, -0.0f, 0.0f, 1.0e-39f, 2.0f, 4.0f, 3.0e38f};
    const float dirs[] = {-1.0f, -0.25f, -1.0e-20f, -2.0e-38f, -1.0e-39f, -1.0e-45f, -0.0f, 0.0f,
                          1.0e-45f, 1.0e-39f, 2.0e-38f, 1.0e-20f, 0.25f, 1.0f, 3.0e38f, inf, -inf, nan};
    std::vector<Axis> axes;
    for (float lo : bounds)
        for (float hi : bounds)
            if (lo <= hi)
                for (float o : origins)
                    for (float d : dirs) {
                        // a tree box is finite or (an empty slot) +infinity on both sides
                        if (std::isinf(d) && std::isinf(lo) != std::isinf(hi)) continue;
                        const float inv = 1.0f / d;
                        axes.push_back({lo, hi, o, d, inv, o * inv});
                    }
    const Axis plain[] = {{-2.0f, 3.0f, 1.0f, 0.5f, 2.0f, 2.0f}, {1.0f, 3.0f, 2.0f, -0.5f, -2.0f, -4.0f}};
    long cases = 0;
    auto check = [&](const Axis& x, const Axis& y, const Axis& z, float tmax) {
        const Axis* a[3] = {&x, &y, &z};
        float n[3], f[3], t0[3], t1[3];
        for (int k = 0; k < 3; k++) {
            const int up = ptg::UpperFirst(a[k]->inv, a[k]->oi);
            n[k] = up ? a[k]->hi : a[k]->lo;
            f[k] = up ? a[k]->lo : a[k]->hi;
            const float p = fmaf(a[k]->lo, a[k]->inv, -a[k]->oi), q = fmaf(a[k]->hi, a[k]->inv, -a[k]->oi);
            t0[k] = fminf(p, q);
            t1[k] = fmaxf(p, q);
        }
        const float got = ptg::SlabEntry(n[0], n[1], n[2], f[0], f[1], f[2], x.inv, y.inv, z.inv, x.oi, y.oi, z.oi, tmax);
        const float tn = fmaxf(fmaxf(t0[0], t0[1]), fmaxf(t0[2], 0.0f));
        const float tf = fminf(fminf(t1[0], t1[1]), fminf(t1[2], tmax));
        const float want = tn <= tf ? tn : inf;
        cases++;
        if (got == want) return true;
        std::printf("differs: got %g want %g\n", got, want);
        for (int k = 0; k < 3; k++)
            std::printf("  axis %d: lo %g hi %g o %g d %g\n", k, a[k]->lo, a[k]->hi, a[k]->o, a[k]->d);
        return false;
    };
    for (const Axis& x : axes)
        for (const Axis& p : plain)
            for (float tmax : {3.4028235e38f, 1.0f, 0.0f}) {
                if (!check(x, p, plain[0], tmax) || !check(p, x, plain[1], tmax) || !check(p, plain[0], x, tmax)) return 1;
            }
    for (size_t i = 0; i < axes.size(); i += 7)
        for (size_t j = 0; j < axes.size(); j += 5)
            if (!check(axes[i], plain[0], axes[j], 3.4028235e38f)) return 1;
    std::printf("ok %ld\n", cases);
    return 0;
}
