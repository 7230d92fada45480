// Device records of a scene (layout in pt_layout.h), formed on the GPU from the caller's
// arrays and the finished BVH (scene_records.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bvh_builder.h"

namespace ptg {

// Device arrays the records are formed from; normals, uvs and shading may be null.
struct SceneArrays {
    const float* positions;      // 3 per vertex
    const float* normals;        // 3 per vertex; null: (0, 0, 1)
    const float* uvs;            // 3 per vertex; null: zero
    const int32_t* indices;      // 3 per triangle
    const int32_t* material;     // per triangle
    const uint8_t* shading;      // per triangle; null: flat
    const int32_t* primIds;      // triangle of each primitive slot
    int numTris;
};

// Records of the binary tree's nodes [first, first + count), given from `in` on: 2 float4 per
// node, and the box word pairs of their slots' triangle records. wideOffset: where the wide tree
// starts, in float4 from `nodes`.
cudaError_t FormNodeRecords(const BvhNodeOut* in, int first, int count, float4* nodes, int wideOffset, float wideEps,
                            float4* tris, cudaStream_t stream);

// tris (but for the box word pairs), shade, uvsOut (may be null): 3 float4 per primitive slot.
cudaError_t FormSlotRecords(const SceneArrays& in, float4* tris, float4* shade, float4* uvsOut, cudaStream_t stream);

// out[i] = {rgb[3 i], rgb[3 i + 1], rgb[3 i + 2], 0} for n texels.
cudaError_t PadTexels(const float* rgb, size_t n, float4* out, cudaStream_t stream);

}  // namespace ptg
