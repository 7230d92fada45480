// What a context's ray queries do beside their launch, over the fake runtime: no work on the
// default stream, which nothing orders with the query's, and the words that tile renders
// report through left alone. Prints "ok" or what differs.
#include <cstdio>

#include "fake_cuda.h"

#include "context.h"
#include "pt_kernels.h"

namespace ptg {
struct Launch {
    int* counter;
    cudaStream_t stream;
    size_t at;  // operations before it
};
static std::vector<Launch> launches;
cudaError_t LaunchTraceClosest(const DevScene&, int, const float*, float, float, int*, float*, int* counter,
                               cudaStream_t stream) {
    launches.push_back({counter, stream, fake::ops.size()});
    return cudaSuccess;
}
void FreeWaveGraphCache(WaveGraphCache*) {}
}  // namespace ptg

#define CHECK(c)                                                 \
    do {                                                         \
        if (!(c)) return std::printf("fails: %s\n", #c), 1;      \
    } while (0)

int main() {
    using namespace ptg;
    pt_context* ctx = nullptr;
    CHECK(pt_context_create(0, 0, &ctx) == PT_OK);
    ctx->scenes[1] = std::make_unique<SceneGpu>();
    const cudaStream_t a = fake::Handle<cudaStream_t>();
    float rays[6] = {}, dist[1];
    int tri[1];
    // the first query of a context, on a stream of the caller's, and one on the context's
    for (void* s : {(void*)a, (void*)nullptr}) {
        fake::ops.clear();
        CHECK(pt_trace_closest(ctx, 1, 1 << 20, rays, 0.0f, 1e30f, tri, dist, s) == PT_OK);
        const cudaStream_t on = s ? (cudaStream_t)s : ctx->stream;
        CHECK(launches.back().stream == on);
        for (const fake::Op& o : fake::ops) CHECK(o.stream == on);
        CHECK(launches.back().counter != nullptr);
        const char* w = (const char*)ctx->status.ptr;
        CHECK(!w || (char*)launches.back().counter < w || (char*)launches.back().counter >= w + ctx->status.bytes);
    }
    CHECK(pt_context_destroy(ctx) == PT_OK);
    CHECK(fake::inUse == 0);
    std::printf("ok\n");
    return 0;
}
