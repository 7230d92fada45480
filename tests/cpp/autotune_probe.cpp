// The autotuner's probe renders over the fake runtime: with probe_spp 0 a probe has at least 4
// samples a pixel, and as many more as make its wave too large for the one launch of small waves
// where the render's is; a probe_spp of the caller's is kept. Prints "ok" or what fails.
#include <algorithm>
#include <cstdio>

#include "fake_cuda.h"

#include "context.h"
#include "pt_kernels.h"

namespace ptg {
static int least = 1 << 30, most = 0;
static size_t Bytes(int capacity) { return 4096 + (size_t)capacity; }
size_t WaveBuffersBytes(int capacity) { return Bytes(capacity); }
size_t WaveBuffersBytesTwoLanes(int capacity) { return 2 * Bytes(capacity); }
WaveBuffers CarveWaveBuffers(void* base, int capacity) {
    WaveBuffers w{};
    w.capacity = capacity;
    w.counts = (int*)base;
    w.ray[0] = (float4*)base;
    return w;
}
WaveGraphCache* NewWaveGraphCache() { return nullptr; }
void FreeWaveGraphCache(WaveGraphCache*) {}
cudaError_t RunWave(const DevJob*, const WaveUnit*, const WaveShape& shape, const WaveBuffers&, cudaStream_t, int*,
                    WaveProfile*, const WaveTuning&, WaveGraphCache*, int, bool) {
    least = std::min(least, shape.nPaths);
    most = std::max(most, shape.nPaths);
    return cudaSuccess;
}
cudaError_t FinalizeJobs(const DevJob*, const int*, int, int, cudaStream_t, int*, WaveProfile*) { return cudaSuccess; }
int WholeWavePaths(bool interior) { return interior ? 70000 : 200000; }
}  // namespace ptg

#define CHECK(c)                                            \
    do {                                                    \
        if (!(c)) return std::printf("fails: %s\n", #c), 1; \
    } while (0)

int main() {
    using namespace ptg;
    struct Case {
        int side, spp, probe, want;
        bool inside;
        int bounces = 8;
    };
    const Case cases[] = {
        {100, 2, 0, 2, false},  {100, 20, 0, 4, false}, {100, 21, 0, 21, false}, {100, 500, 0, 21, false},
        {100, 500, 3, 3, false}, {300, 64, 0, 4, false}, {100, 64, 0, 8, true},   {100, 7, 0, 4, true},
        {100, 64, 0, 21, true, 3}, {1, 1 << 20, 0, 200001, false}};
    for (const Case& c : cases) {
        pt_context* ctx = nullptr;
        CHECK(pt_context_create(0, 0, &ctx) == PT_OK);
        auto sg = std::make_unique<SceneGpu>();
        for (int a = 0; a < 3; a++) sg->lo[a] = -1.0f, sg->hi[a] = 1.0f;
        sg->dev.numTris = 12;
        sg->dev.numLights = 1;
        ctx->scenes[1] = std::move(sg);
        pt_camera cam{};
        cam.pos[0] = c.inside ? 0.5f : 5.0f;
        pt_settings st{};
        st.width = st.height = c.side;
        st.spp = c.spp;
        st.max_bounces = c.bounces;
        st.tile_width = st.tile_height = 1;
        st.integrator = PT_INTEGRATOR_PT;
        st.mode = PT_MODE_WAVEFRONT;
        least = 1 << 30;
        most = 0;
        CHECK(pt_autotune(ctx, 1, &cam, &st, c.probe, nullptr) == PT_OK);
        if (least != most || most != c.side * c.side * c.want)
            return std::printf("%d x %d x %d: probes of %d to %d paths\n", c.side, c.side, c.spp, least, most), 1;
        CHECK(pt_context_destroy(ctx) == PT_OK);
    }
    std::printf("ok\n");
    return 0;
}
