// Device binned-SAH BVH build (bvh_gpu.cu): the tree of BuildBinnedSah, built on the GPU.
#pragma once
#include <cuda_runtime.h>

#include <string>

#include "bvh_builder.h"

namespace ptg {

struct DeviceBuildStats {
    double ms = 0.0;  // device time from the first copy to the tree read back
    int levels = 0, rounds = 0, heapsorts = 0, launches = 0;
};

// A build's device arrays, kept for the caller: all in one allocation, to be freed with
// cudaFree(block). Its other arrays are done with: their bytes are the caller's to use.
struct DeviceBvh {
    void* block = nullptr;
    const float* positions = nullptr;
    const int32_t* indices = nullptr;
    const BvhNodeOut* nodes = nullptr;
    const int32_t* primIds = nullptr;
    char* spare = nullptr;  // on a 256-byte boundary
    size_t spareBytes = 0;
};

// positions: numVertices x 3 floats, indices: numTriangles x 3 (host memory, validated
// by the caller). Allocates its scratch (398 bytes per triangle and 12 per vertex) for the
// build in one piece and frees it, or hands it to `keep` (null: not kept; left alone when there are
// no triangles); synchronises `stream`. On failure `out` is empty and `error` says why.
cudaError_t BuildBinnedSahDevice(const float* positions, int numVertices, const int32_t* indices,
                                 int numTriangles, cudaStream_t stream, BvhResult* out,
                                 std::string* error, DeviceBuildStats* stats, DeviceBvh* keep = nullptr);

}  // namespace ptg
