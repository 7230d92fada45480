// Which waves count as interiors (csrc/scheduler.h ShapeOf): most paths of jobs with the camera
// inside and area lights, in waves of fixed depth. Prints "ok" or the first difference.
#include <cstdio>
#include <vector>

#include "scheduler.h"

static ptg::DevJob Job(int side, int inside, int lights, int integrator, int bounces = 4) {
    ptg::DevJob J{};
    J.st.width = J.st.height = side;
    J.st.spp = 1;
    J.st.maxBounces = bounces;
    J.st.integrator = integrator;
    J.S.numTris = 100;
    J.S.numLights = lights;
    J.inside = inside;
    return J;
}

int main() {
    using namespace ptg;
    struct Case {
        std::vector<DevJob> jobs;
        int want;
    };
    const std::vector<Case> cases = {
        {{Job(8, 1, 2, kPathTracing)}, 1},
        {{Job(8, 0, 2, kPathTracing)}, 0},
        {{Job(8, 1, 2, kPathTracing, 3)}, 0},  // few bounces
        {{Job(8, 1, 0, kPathTracing)}, 0},
        {{Job(8, 1, 2, kSimplePathTracing)}, 0},  // ends where its queue does
        {{Job(8, 1, 2, kPathTracing), Job(7, 0, 2, kPathTracing)}, 1},
        {{Job(8, 1, 2, kPathTracing), Job(8, 0, 2, kPathTracing)}, 0},
        {{Job(8, 0, 0, kPathTracing), Job(9, 1, 1, kPathTracing)}, 1},
    };
    for (size_t k = 0; k < cases.size(); k++) {
        std::vector<std::vector<WaveUnit>> waves;
        if (!PlanWaves(cases[k].jobs, 1 << 20, 64, &waves) || waves.size() != 1) return std::printf("no plan\n"), 1;
        const WaveShape s = ShapeOf(cases[k].jobs, waves[0], 0);
        if (s.interior != cases[k].want) return std::printf("case %zu: %d\n", k, s.interior), 1;
    }
    std::printf("ok\n");
    return 0;
}
