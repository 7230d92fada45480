// A context's first wavefront renders on a caller's stream, over the fake runtime: the wave
// buffers it allocates are cleared on that stream and on no other, which nothing orders with
// the wave's kernels. Prints "ok" or what differs.
#include <cstdio>

#include "fake_cuda.h"

#include "context.h"
#include "pt_kernels.h"

namespace ptg {
static cudaStream_t waveStream;
static int waves = 0;
static size_t Bytes(int capacity) { return 4096 + 64 * (size_t)capacity; }
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
cudaError_t RunWave(const DevJob*, const WaveUnit*, const WaveShape&, const WaveBuffers&, cudaStream_t s, int*, WaveProfile*,
                    const WaveTuning&, WaveGraphCache*, int, bool) {
    waveStream = s;
    waves++;
    return cudaSuccess;
}
cudaError_t FinalizeJobs(const DevJob*, const int*, int, int, cudaStream_t, int*, WaveProfile*) { return cudaSuccess; }
}  // namespace ptg

#define CHECK(c)                                            \
    do {                                                    \
        if (!(c)) return std::printf("fails: %s\n", #c), 1; \
    } while (0)

int main() {
    using namespace ptg;
    pt_context* ctx = nullptr;
    CHECK(pt_context_create(0, 0, &ctx) == PT_OK);
    ctx->scenes[1] = std::make_unique<SceneGpu>();
    const cudaStream_t a = fake::Handle<cudaStream_t>();
    pt_camera cam{};
    cam.h_perf = 1.0f;
    pt_settings st{};
    st.spp = st.tile_width = st.tile_height = 1;
    st.integrator = PT_INTEGRATOR_PT;
    st.mode = PT_MODE_WAVEFRONT;
    float film[3 * 64];
    for (int side : {4, 8}) {  // the second render grows the buffers
        st.width = st.height = side;
        fake::ops.clear();
        CHECK(pt_render_device(ctx, 1, &cam, &st, film, a) == PT_OK);
        CHECK(waveStream == a);
        const char* lo = (const char*)ctx->wbBuffers[0].ptr;
        bool cleared = false;
        for (const fake::Op& o : fake::ops)
            if ((const char*)o.what >= lo && (const char*)o.what < lo + ctx->wbBuffers[0].bytes) {
                CHECK(o.stream == a);
                cleared |= o.kind == fake::Op::kSet && o.what == ctx->wb.counts;
            }
        CHECK(cleared);
    }
    CHECK(waves == 2);
    // buffers that could not grow are gone: nothing reads the freed ones
    st.width = st.height = 1024;
    fake::limit = fake::inUse;
    CHECK(pt_render_device(ctx, 1, &cam, &st, film, a) == PT_ERR_OUT_OF_MEMORY);
    CHECK(ctx->wb.counts == nullptr || fake::blocks.count(ctx->wbBuffers[0].ptr));
    fake::limit = 0;
    st.width = st.height = 8;
    CHECK(pt_render_device(ctx, 1, &cam, &st, film, a) == PT_OK && waves == 3);
    CHECK(pt_context_destroy(ctx) == PT_OK && fake::inUse == 0);
    std::printf("ok\n");
    return 0;
}
