// Device memory of a scene upload over the fake runtime, with the host builder, and with it
// standing in for the device build (which takes and keeps a block as that one does). An
// upload with room for the larger of the build and the scene (host builder: the scene and a
// step's sources), and for one part of an image, is accepted with the records of one that had
// all the room; with less than the scene it is refused. Prints "ok" or
// what fails.
#include <cstdio>
#include <functional>

#include "fake_cuda.h"

#include "bvh_gpu.h"
#include "context.h"
#include "scene_records.h"

namespace ptg {
constexpr size_t kKept = 110, kBuild = 398;  // bytes a triangle: kept arrays, all arrays
static size_t Up(size_t b) { return (b + 255) & ~size_t(255); }

cudaError_t BuildBinnedSahDevice(const float* pos, int nv, const int32_t* idx, int T, cudaStream_t, BvhResult* out,
                                 std::string* error, DeviceBuildStats*, DeviceBvh* keep) {
    const size_t need = kBuild * T + 12 * (size_t)nv + 1024;
    void* block = nullptr;
    if (cudaMalloc(&block, need) != cudaSuccess) return *error = "device BVH build: allocation failed", cudaErrorMemoryAllocation;
    *out = BuildBinnedSah(pos, idx, T, 1);
    char* p = (char*)block;
    auto put = [&](const void* from, size_t bytes) {
        char* at = p;
        std::memcpy(at, from, bytes);
        p += Up(bytes);
        return (void*)at;
    };
    keep->block = block;
    keep->positions = (float*)put(pos, 12 * (size_t)nv);
    keep->indices = (int32_t*)put(idx, 12 * (size_t)T);
    keep->nodes = (BvhNodeOut*)put(out->nodes.data(), out->nodes.size() * sizeof(BvhNodeOut));
    keep->primIds = (int32_t*)put(out->primIds.data(), 4 * (size_t)T);
    keep->spare = p;
    keep->spareBytes = (size_t)((char*)block + need - p);
    return cudaSuccess;
}
// Records that hold every word their kernels read.
cudaError_t FormNodeRecords(const BvhNodeOut* in, int first, int count, float4* nodes, int wideOffset, float eps, float4* tris,
                            cudaStream_t) {
    for (int i = 0; i < count; i++) {
        const BvhNodeOut& n = in[i];
        nodes[2 * (size_t)(first + i)] = float4{n.lo[0], n.lo[1], n.lo[2], n.hi[0]};
        nodes[2 * (size_t)(first + i) + 1] = float4{n.hi[1], n.hi[2], (float)(n.leaf ? n.begin : n.child[0]), (float)n.end};
        for (int k = n.begin; n.leaf && k < n.end; k++) {
            tris[3 * (size_t)k + 2].z = (float)(2 * (first + i) - wideOffset);
            tris[3 * (size_t)k + 2].w = eps;
        }
    }
    return cudaGetLastError();
}
cudaError_t FormSlotRecords(const SceneArrays& in, float4* tris, float4* shade, float4* uvs, cudaStream_t) {
    for (int k = 0; k < in.numTris; k++) {
        const int t = in.primIds[k];
        for (int v = 0; v < 3; v++) {
            const float* x[3] = {in.positions, in.normals, in.uvs};
            const size_t at = 3 * (size_t)in.indices[3 * t + v];
            for (int a = 0; a < 3; a++) {
                (&tris[3 * (size_t)k].x)[3 * v + a] = x[0][at + a];
                (&shade[3 * (size_t)k].x)[3 * v + a] = x[1][at + a];
                if (uvs) (&uvs[3 * (size_t)k].x)[3 * v + a] = x[2][at + a];
            }
        }
        shade[3 * (size_t)k + 2].y = (float)in.material[t];
        shade[3 * (size_t)k + 2].z = (float)in.shading[t];
    }
    return cudaGetLastError();
}
cudaError_t PadTexels(const float* rgb, size_t n, float4* out, cudaStream_t) {
    for (size_t i = 0; i < n; i++) out[i] = float4{rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], 0.0f};
    return cudaGetLastError();
}
cudaError_t FillEnvTable(const DevScene&, float4*, cudaStream_t) { return cudaGetLastError(); }
cudaError_t FillEnvTableExact(const DevScene&, float4*, cudaStream_t) { return cudaGetLastError(); }
void FreeWaveGraphCache(WaveGraphCache*) {}
}  // namespace ptg

#define CHECK(c)                                                                         \
    do {                                                                                 \
        if (!(c)) return std::printf("fails for %s: %s (%s)\n", name, #c, pt_last_error(ctx)), 1; \
    } while (0)

int main() {
    using namespace ptg;
    struct Case {
        const char* name;
        int tris, env, maps, mapSide;
        bool indexed;
    };
    const Case cases[] = {{"mesh", 30000, 0, 0, 0, true},       {"loose triangles", 20000, 16, 0, 0, false},
                          {"mesh and sky", 9000, 700, 0, 0, true}, {"sky alone", 0, 900, 0, 0, true},
                          {"maps", 5000, 32, 9, 160, true},     {"few triangles", 36, 512, 1, 300, false}};
    for (int builder : {PT_BVH_BUILDER_DEVICE, PT_BVH_BUILDER_HOST})
    for (const Case& c : cases) {
        const char* name = c.name;
        const int T = c.tris, side = 1 + T / 2, nv = c.indexed ? side + 3 : 3 * T;
        auto value = [](size_t i) { return (float)((i * 2654435761u >> 7) % 1009) / 64.0f; };
        std::vector<float> pos(3 * (size_t)nv), nrm(3 * (size_t)nv), uv(3 * (size_t)nv);
        for (size_t i = 0; i < pos.size(); i++) pos[i] = value(i), nrm[i] = value(i + 5), uv[i] = value(3 * i + 1);
        std::vector<int32_t> idx(3 * (size_t)T), mat(T);
        std::vector<uint8_t> sh(T);
        for (int t = 0; t < T; t++) {
            for (int v = 0; v < 3; v++) idx[3 * (size_t)t + v] = c.indexed ? (t / 2 + v) : 3 * t + v;
            mat[t] = t % 3;
            sh[t] = t & 1;
        }
        std::vector<float> sky(3 * (size_t)c.env * (c.env / 2)), map(3 * (size_t)c.mapSide * c.mapSide);
        for (size_t i = 0; i < sky.size(); i++) sky[i] = value(i);
        for (size_t i = 0; i < map.size(); i++) map[i] = value(7 * i);
        std::vector<pt_texture> tex(c.maps);
        for (pt_texture& x : tex) x.width = x.height = c.mapSide, x.rgb = map.data();
        pt_material mats[3] = {};
        for (pt_material& m : mats) m.kind = PT_MAT_LAMBERT, m.tex_albedo = c.maps ? 1 : 0;
        pt_scene_desc d{};
        d.num_vertices = nv;
        d.num_triangles = T;
        d.positions = pos.data();
        d.normals = nrm.data();
        d.uvs = c.maps || !c.indexed ? uv.data() : nullptr;
        d.indices = idx.data();
        d.tri_material = mat.data();
        d.tri_shading = sh.data();
        d.num_materials = 3;
        d.materials = mats;
        d.env_width = c.env;
        d.env_height = c.env / 2;
        d.env_rgb = c.env ? sky.data() : nullptr;
        d.num_textures = c.maps;
        d.textures = tex.data();
        pt_context* ctx = nullptr;
        CHECK(pt_context_create(0, 0, &ctx) == PT_OK && pt_set_bvh_builder(ctx, builder) == PT_OK);
        const bool device = builder == PT_BVH_BUILDER_DEVICE;
        const size_t sources = 36 * (size_t)nv + 21 * (size_t)T;
        const size_t build = T && device ? kBuild * T + 12 * (size_t)nv + 1024 : 0;
        std::vector<std::vector<char>> want;
        size_t scene = 0;
        // all the room, then the least an upload may ask for, then less than the scene
        for (int round = 0; round < 3; round++) {
            const size_t part = size_t(64) << 10;
            fake::limit = round == 0 ? 0 : round == 1 ? std::max(build, scene + (device ? 0 : sources)) + part : scene - 1;
            pt_scene_id id = 0;
            const int rc = pt_scene_upload(ctx, &d, &id);
            if (round == 2) {
                CHECK(rc == PT_ERR_OUT_OF_MEMORY && fake::inUse == 0);
                break;
            }
            CHECK(rc == PT_OK);
            if (round == 0) scene = fake::inUse;
            const DevScene& S = ctx->scenes[id]->dev;
            for (size_t i = 0; i < sky.size() / 3; i++) CHECK(S.env[i].x == sky[3 * i] && S.env[i].z == sky[3 * i + 2]);
            for (int t = 0; t < c.maps; t++)
                for (size_t i = 0; i < map.size() / 3; i++) CHECK(S.texels[S.texInfo[t].x + i].y == map[3 * i + 1]);
            CHECK(fake::inUse == scene);
            std::vector<std::vector<char>> got;
            const float4* records[] = {S.nodes, S.tris, S.shade, S.uvs};
            for (int r = 0; r < 4; r++) {
                const size_t n = !records[r] ? 0 : 16 * (r == 0 ? (size_t)(S.wide - S.nodes) : 3 * (size_t)T);
                got.emplace_back((const char*)records[r], (const char*)records[r] + n);
            }
            if (round == 0) want = got;
            CHECK(got == want);
            CHECK(pt_scene_release(ctx, id) == PT_OK && fake::inUse == 0);
        }
        fake::limit = 0;
        CHECK(pt_context_destroy(ctx) == PT_OK && fake::inUse == 0);
    }
    std::printf("ok\n");
    return 0;
}
