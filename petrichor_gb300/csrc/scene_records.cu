// Scene records formed on the GPU. They were formed on the host's cores and copied up:
// 112 MB of freshly paged vectors for 400,000 triangles and a 1024x512 sky, 9 ms of a 27.6 ms
// upload. Here the caller's arrays go up as they are (or are there already from the BVH build)
// and one thread per slot forms its records with the same float operations; bound by HBM
// writes (144 bytes a triangle). Upload of 20,000 / 400,000 / 1.0M triangles: 5.3 / 25.0 / 51.4
// ms -> 3.8 / 15.2 / 27.4 ms (with the build's arrays in one allocation).
#include "scene_records.h"

#include "pt_layout.h"

namespace ptg {
namespace {

constexpr int kThreads = 256;
constexpr int kOwnSlots = 64;  // a leaf's slots its own thread marks; longer leaves take the warp

// A primitive slot's last word pair: {box, eps} of its triangle record.
__device__ __forceinline__ void MarkBox(float4* tris, int slot, int node, int wideOffset, float eps) {
    float* w = reinterpret_cast<float*>(tris + 3 * (size_t)slot + 2);
    w[2] = __int_as_float(2 * node - wideOffset);
    w[3] = eps;
}

__global__ void __launch_bounds__(kThreads) NodeRecords(const BvhNodeOut* __restrict__ in, int first, int count,
                                                        float4* __restrict__ nodes, int wideOffset, float wideEps,
                                                        float4* __restrict__ tris) {
    const int at = blockIdx.x * kThreads + threadIdx.x;
    const int i = first + at;
    const int lane = threadIdx.x & 31;
    int begin = 0, end = 0;
    if (at < count) {
        const BvhNodeOut n = in[at];
        nodes[2 * (size_t)i] = make_float4(n.lo[0], n.lo[1], n.lo[2], n.hi[0]);
        nodes[2 * (size_t)i + 1] = make_float4(n.hi[1], n.hi[2], __int_as_float(n.leaf ? n.begin : n.child[0]),
                                               __int_as_float(n.leaf ? n.end - n.begin : -1));
        if (n.leaf) begin = n.begin, end = n.end;
    }
    const bool big = end - begin > kOwnSlots;
    if (!big)
        for (int k = begin; k < end; k++) MarkBox(tris, k, i, wideOffset, wideEps);
    for (unsigned m = __ballot_sync(0xffffffffu, big); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int b = __shfl_sync(0xffffffffu, begin, j), e = __shfl_sync(0xffffffffu, end, j);
        for (int k = b + lane; k < e; k += 32) MarkBox(tris, k, i - lane + j, wideOffset, wideEps);
    }
}

__global__ void __launch_bounds__(kThreads) SlotRecords(SceneArrays in, float4* __restrict__ tris,
                                                        float4* __restrict__ shade, float4* __restrict__ uvsOut) {
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= in.numTris) return;
    const int t = in.primIds[k];
    float p[3][3], n[3][3] = {{0, 0, 1}, {0, 0, 1}, {0, 0, 1}};
    for (int v = 0; v < 3; v++) {
        const size_t x = 3 * (size_t)in.indices[3 * (size_t)t + v];
        for (int a = 0; a < 3; a++) {
            p[v][a] = in.positions[x + a];
            if (in.normals) n[v][a] = in.normals[x + a];
        }
        if (uvsOut)
            uvsOut[3 * (size_t)k + v] =
              in.uvs ? make_float4(in.uvs[x], in.uvs[x + 1], in.uvs[x + 2], 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float e1[3], e2[3];
    for (int a = 0; a < 3; a++) {
        e1[a] = p[1][a] - p[0][a];
        e2[a] = p[2][a] - p[0][a];
    }
    tris[3 * (size_t)k] = make_float4(p[0][0], p[0][1], p[0][2], e1[0]);
    tris[3 * (size_t)k + 1] = make_float4(e1[1], e1[2], e2[0], e2[1]);
    float* last = reinterpret_cast<float*>(tris + 3 * (size_t)k + 2);  // its other half is NodeRecords'
    last[0] = e2[2];
    last[1] = __int_as_float(t);
    const int smooth = in.shading && in.shading[t] ? 1 : 0;
    shade[3 * (size_t)k] = make_float4(n[0][0], n[0][1], n[0][2], __int_as_float(in.material[t]));
    shade[3 * (size_t)k + 1] = make_float4(n[1][0], n[1][1], n[1][2], __int_as_float(smooth));
    shade[3 * (size_t)k + 2] = make_float4(n[2][0], n[2][1], n[2][2], 0.0f);
}

__global__ void __launch_bounds__(kThreads) PadKernel(const float* __restrict__ rgb, size_t n, float4* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
    if (i < n) out[i] = make_float4(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], 0.0f);
}

unsigned Blocks(size_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

}  // namespace

cudaError_t FormNodeRecords(const BvhNodeOut* in, int first, int count, float4* nodes, int wideOffset, float wideEps,
                            float4* tris, cudaStream_t stream) {
    if (count > 0)
        NodeRecords<<<Blocks(count), kThreads, 0, stream>>>(in, first, count, nodes, wideOffset, wideEps, tris);
    return cudaGetLastError();
}

cudaError_t FormSlotRecords(const SceneArrays& in, float4* tris, float4* shade, float4* uvsOut, cudaStream_t stream) {
    if (in.numTris > 0) SlotRecords<<<Blocks(in.numTris), kThreads, 0, stream>>>(in, tris, shade, uvsOut);
    return cudaGetLastError();
}

cudaError_t PadTexels(const float* rgb, size_t n, float4* out, cudaStream_t stream) {
    if (n > 0) PadKernel<<<Blocks(n), kThreads, 0, stream>>>(rgb, n, out);
    return cudaGetLastError();
}

}  // namespace ptg
