// What a context's ray queries do beside their launch, over the fake runtime: no work on the
// default stream, which nothing orders with the query's, and the words that tile renders
// report through left alone; and a counter that no other query that may still run uses,
// whatever their streams, captured or not. Prints "ok" or what differs.
#include <cstdio>

#include "fake_cuda.h"

#include "context.h"
#include "pt_kernels.h"

namespace ptg {
static bool longQueries = true;
bool TraceUsesCounter(int) { return longQueries; }
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
    // queries on several streams: a counter is used again only behind the query that had it
    const cudaStream_t streams[] = {a, fake::Handle<cudaStream_t>(), fake::Handle<cudaStream_t>()};
    std::map<int*, cudaEvent_t> last;  // counter -> recorded behind its latest query
    fake::ops.clear();
    launches.clear();
    size_t seen = 0;
    for (int k = 0; k < 200; k++) {
        const cudaStream_t s = streams[(k * 7 / 3) % 3];
        CHECK(pt_trace_closest(ctx, 1, 1 << 20, rays, 0.0f, 1e30f, tri, dist, s) == PT_OK);
        const Launch& l = launches.back();
        if (last.count(l.counter)) {
            bool waited = false;
            for (size_t i = seen; i < l.at; i++)
                waited |= fake::ops[i].kind == fake::Op::kWait && fake::ops[i].stream == s &&
                          fake::ops[i].what == last[l.counter];
            CHECK(waited);
        }
        const fake::Op& end = fake::ops.back();
        CHECK(end.kind == fake::Op::kRecord && end.stream == s && fake::ops.size() == l.at + 1);
        last[l.counter] = (cudaEvent_t)end.what;
        seen = fake::ops.size();
    }
    CHECK(last.size() >= 8);
    // captured queries use no event of the others and none of their counters
    fake::capturing.insert(a);
    std::set<int*> captured;
    fake::ops.clear();
    for (int k = 0; k < 8; k++) {
        CHECK(pt_trace_closest(ctx, 1, 1 << 20, rays, 0.0f, 1e30f, tri, dist, a) == PT_OK);
        CHECK(!last.count(launches.back().counter));
        captured.insert(launches.back().counter);
    }
    CHECK(captured.size() == 8 && fake::ops.empty());
    fake::capturing.clear();
    // short queries need neither
    longQueries = false;
    CHECK(pt_trace_closest(ctx, 1, 10, rays, 0.0f, 1e30f, tri, dist, a) == PT_OK);
    CHECK(launches.back().counter == nullptr && fake::ops.empty());
    CHECK(pt_context_destroy(ctx) == PT_OK);
    CHECK(fake::inUse == 0);
    std::printf("ok\n");
    return 0;
}
