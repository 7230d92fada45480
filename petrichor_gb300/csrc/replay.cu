// Replay kernel: reproduces the reference renderer's film bit for bit.
//
// The reference draws its random numbers from one XorShift stream per 16x16
// tile, visiting the tile's pixels row-major (Core/Petrichor.cpp:79-91), so a
// pixel's samples depend on every earlier pixel of its tile. This kernel runs
// one warp per tile with that stream, the reference's BVH traversal order and
// the reference's arithmetic (ExactMath, built with -fmad=false). It is the
// parity path; the wavefront kernels are the throughput path.
//
// A tile is one serial chain, so the kernels are bound by its latency: the traversal's
// node steps and triangle tests first, then the FP64 functions (1400-2600 cycles each).
// The 32 lanes of a tile's warp run the same path on the same values and split the work
// inside a traversal (TraverseWarp): the two children of a node, and a leaf's triangles,
// are tested side by side. FP64 costs a warp the same with one active lane or 32.
// One thread per tile, 32 diverging tiles to a warp, took 173.4 ms for a 256x256 2-spp
// Cornell box and 111.6 ms for a 960x540 4-spp albedo pass over 200,000 triangles; one
// active lane per warp 39.5 and 40.8 ms; this form 33.6 and 35.0 ms (passes on several streams
// overlap: 16.6 and 16.7-23.8 ms each).
#include <cuda_runtime.h>

#include "pt_device.cuh"
#include "pt_kernels.h"

namespace ptg {

// Entries of a warp's traversal stack in shared memory; deeper ones keep the node index
// alone in the tile's scratch.
constexpr int kReplaySmemStack = 24;

struct WarpStack {
    int4* near;  // shared: {first, count, entry distance bits, origin inside}
    int* deep;   // global: node index
};

// One node of the reference's traversal (TraverseReference): whether the ray passes the
// slab test, the distance the node is culled by and whether the origin lies inside it.
struct NodeTest {
    bool pass, inside;
    int a, cnt;
    float nd, centre;  // centre: squared distance of the box centre from the origin
};
__device__ __forceinline__ NodeTest TestNode(const float4* __restrict__ nodes, int ni, V3 o, V3 inv) {
    const float4 na = __ldg(nodes + 2 * ni), nb = __ldg(nodes + 2 * ni + 1);
    const V3 lo(na.x, na.y, na.z), hi(na.w, nb.x, nb.y);
    NodeTest r;
    r.a = __float_as_int(nb.z);
    r.cnt = __float_as_int(nb.w);
    const bool s0 = inv.x < 0.0f, s1 = inv.y < 0.0f, s2 = inv.z < 0.0f;
    float tMin = __fmul_rn((s0 ? hi : lo).x - o.x, inv.x);
    float tMax = __fmul_rn((s0 ? lo : hi).x - o.x, inv.x);
    const float tyMin = __fmul_rn((s1 ? hi : lo).y - o.y, inv.y);
    const float tyMax = __fmul_rn((s1 ? lo : hi).y - o.y, inv.y);
    const bool missY = tyMax < tMin || tMax < tyMin;
    if (tMin < tyMin) tMin = tyMin;
    if (tyMax < tMax) tMax = tyMax;
    const float tzMin = __fmul_rn((s2 ? hi : lo).z - o.z, inv.z);
    const float tzMax = __fmul_rn((s2 ? lo : hi).z - o.z, inv.z);
    const bool missZ = tzMax < tMin || tMax < tzMin;
    if (tMin < tzMin) tMin = tzMin;
    if (tzMax < tMax) tMax = tzMax;
    r.nd = kFltMax;
    const bool nearOk = (0.0f <= tMin && tMin < r.nd);
    if (nearOk) r.nd = tMin;
    const bool farOk = (0.0f <= tMax && tMax < r.nd);
    if (farOk) r.nd = tMax;
    r.pass = !missY && !missZ && (nearOk || farOk);
    r.inside = lo.x < o.x && o.x < hi.x && lo.y < o.y && o.y < hi.y && lo.z < o.z &&
               o.z < hi.z;  // AABB::Contains
    r.centre = SqLenRn(CentreRn(lo, hi) - o);
    return r;
}

// TraverseReference by a whole warp for one ray (the same arguments in every lane): the
// same nodes' tests, culls and triangle tests in the same order, so the same answer. A
// node's test does not depend on the hits so far; only the cull against the nearest one
// does, and that is made when the node's turn comes.
//   inner node: even lanes test the left child, odd lanes the right one; the nearer one
//               (by box centre) is next if it passes, the other goes on the stack;
//   leaf:       lane k tests triangle k (32 at a time), the hits are then taken in order.
__device__ int TraverseWarp(const DevScene& S, V3 o, V3 d, float distMin, float distMax, float& bestD,
                            const WarpStack& stk, int* status) {
    if (S.numNodes == 0) return -1;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const V3 inv = ExactRecip(d);
    int sp = 0, best = -1;
    bestD = kInfinity;
    NodeTest cur = TestNode(S.nodes, 0, o, inv);
    bool have = cur.pass;
    for (;;) {
        if (!have) {
            if (sp == 0) break;
            sp--;
            if (sp < kReplaySmemStack) {
                const int4 e = stk.near[sp];
                cur.a = e.x;
                cur.cnt = e.y;
                cur.nd = __int_as_float(e.z);
                cur.inside = e.w != 0;
            } else {
                cur = TestNode(S.nodes, stk.deep[sp], o, inv);
            }
            have = !(best >= 0 && !cur.inside && bestD < cur.nd);
            continue;
        }
        if (PT_CHECK && (cur.cnt >= 0 ? (cur.a < 0 || cur.a + cur.cnt > S.numTris)
                                      : (cur.a < 0 || cur.a + 1 >= S.numNodes))) {
            *status |= kErrBounds;
            return best;
        }
        if (cur.cnt >= 0) {
            for (int k0 = 0; k0 < cur.cnt; k0 += 32) {
                const int k = cur.a + k0 + lane;
                float t = 0.0f;
                bool hit = false;
                if (k0 + lane < cur.cnt) {
                    V3 v0, e1, e2;
                    LoadTri(S.tris, k, v0, e1, e2);
                    hit = TriIntersect(v0, e1, e2, o, d, t) && !(t < distMin || t > distMax);
                }
                for (unsigned m = __ballot_sync(kAll, hit); m; m &= m - 1) {
                    const int j = __ffs(m) - 1;
                    const float tj = __shfl_sync(kAll, t, j);
                    if (best < 0 || tj < bestD) {
                        best = cur.a + k0 + j;
                        bestD = tj;
                    }
                }
            }
            have = false;
        } else {
            const int side = lane & 1;
            const NodeTest c = TestNode(S.nodes, cur.a + side, o, inv);
            const bool alive = c.pass && !(best >= 0 && !c.inside && bestD < c.nd);
            const unsigned up = __ballot_sync(kAll, alive);
            const float other = __shfl_xor_sync(kAll, c.centre, 1);
            // the left child first when its centre is nearer
            const bool mineFirst = side ? !(other < c.centre) : c.centre < other;
            const int first = __ffs(__ballot_sync(kAll, mineFirst)) - 1;  // 0 or 1
            if (sp + 1 > S.stackDepth) {
                *status |= kErrStackOverflow;
                return best;
            }
            if (up >> (first ^ 1) & 1) {
                if (sp < kReplaySmemStack) {
                    if (lane == (first ^ 1))
                        stk.near[sp] = make_int4(c.a, c.cnt, __float_as_int(c.nd), c.inside ? 1 : 0);
                } else if (lane == (first ^ 1)) {
                    stk.deep[sp] = cur.a + side;
                }
                sp++;
                __syncwarp();
            }
            have = up >> first & 1;
            if (have) {
                cur.a = __shfl_sync(kAll, c.a, first);
                cur.cnt = __shfl_sync(kAll, c.cnt, first);
            }
        }
    }
    return best;
}

__device__ __forceinline__ bool IsEmission(const DevScene& S, int m) { return S.mats[m].kind == kEmission; }

// SimplePathTracing::Render (Core/Integrator/SimplePathTracing.cpp:16-101)
__device__ void ReplaySimplePixel(const DevScene& S, const DevCamera& C, const DevSettings& st,
                                  int px, int py, float* film, RefSampler1D& s1, RefSampler2D& s2,
                                  const WarpStack& stack, int* status) {
    V3 sum;
    for (int sp = 0; sp < st.spp; sp++) {
        float r0, r1, r2, r3;
        s2.Next(r0, r1);
        s2.Next(r2, r3);
        Ray ray = GenerateRay<ExactMath>(C, px, py, st.width, st.height, r0, r1, r2, r3);
        V3 contrib;
        for (int guard = 0;; guard++) {
            if (guard >= kMaxReplayBounces) {  // never reached by terminating paths; see header
                *status |= kErrBounceCap;
                break;
            }
            float dist;
            const int k = TraverseWarp(S, ray.o, ray.d, kEps, kInfinity, dist, stack, status);
            if (k < 0) {
                contrib = contrib + ray.T * EnvColor<ExactMath>(S, ray.d);
                break;
            }
            const int m = ResolveMaterial(S.mats, SlotMaterial(S.shade, k), s1.Next());
            if (IsEmission(S, m)) {
                contrib = contrib + ray.T * MatColor(S.mats[m]);
                break;
            }
            Shading si = Interpolate<ExactMath>(S, k, ray.o, ray.d, dist);
            DevMaterial Mh;
            si.n = PointMaterial<ExactMath>(S, m, k, ray.o, ray.d, si.n, Mh);
            ray = NextRay<ExactMath>(Mh, ray, si, s2);
            if (ray.bounce > st.maxBounces) {
                ray.prob *= 0.9f;
                ray.prob = SMax(0.1f, ray.prob);
                if (s1.Next() < ray.prob) ray.T = ray.T / ray.prob;
                else break;
            }
        }
        sum = sum + contrib;
    }
    const V3 avg = sum / (float)st.spp;
    if ((threadIdx.x & 31) == 0) {
        float* o = film + ((size_t)py * st.width + px) * 3;
        o[0] = avg.x;
        o[1] = avg.y;
        o[2] = avg.z;
    }
}

// PathTracing::SampleLight (PathTracing.cpp:329-386): picks index, samples every
// light (one 2D draw each, as the reference does) and keeps the picked point.
__device__ V3 ReplaySampleLight(const DevScene& S, float rv, RefSampler2D& s2, bool wantEnv,
                                bool* sampleEnv) {
    const int L = S.numLights;
    int index;
    if (!wantEnv) {
        index = (int)(rv * (float)L);
        index = min(index, L - 1);
    } else {
        index = (int)(rv * (float)(L + 1));
        index = min(index, L);
        if (index >= L) {
            *sampleEnv = true;
            return V3();
        }
    }
    V3 result;
    for (int i = 0; i < L; i++) {
        float u0, u1;
        s2.Next(u0, u1);
        const V3 p = SampleLightPoint<ExactMath>(S, i, u0, u1);
        if (i == index) result = p;
    }
    return result;
}

// PathTracing::CalcLightContribution (PathTracing.cpp:202-327)
// M and nb: the shading point's material and BSDF normal (texture maps applied)
__device__ V3 ReplayLight(const DevScene& S, const Shading& si, const DevMaterial& M, V3 nb,
                          RefSampler1D& s1, RefSampler2D& s2, const Ray& ray,
                          const WarpStack& stack, int* status) {
    V3 lc;
    const float dt = -Dot(ray.d, si.n);
    const V3 p = si.pos + kEps * copysignf(1.0f, dt) * si.n;
    const float pdfArea = S.lightPdfArea;
    bool sampleEnv = false;
    const V3 pl = ReplaySampleLight(S, s1.Next(), s2, true, &sampleEnv);
    if (!sampleEnv) {
        if (S.numLights == 0) return V3();
        const V3 ld = Normalized(pl - p);
        float d;
        const int k = TraverseWarp(S, p, ld, 0.0f, kFltMax, d, stack, status);
        if (k >= 0) {
            if (IsEmission(S, ResolveMaterial(S.mats, SlotMaterial(S.shade, k), s1.Next()))) {
                const Shading sl = Interpolate<ExactMath>(S, k, p, ld, d);
                const float dist = SqLen(pl - sl.pos);
                if (fabsf(dist - 0.0f) < kEps) {
                    const float l2 = SqLen(sl.pos - si.pos);
                    const float cosP = fabsf(Dot(ld, sl.n));
                    float mis = 0.0f;
                    if (l2 > 0.0f) {
                        const float pL = pdfArea;
                        const float pB = BsdfPdf<ExactMath>(M, ray.d, ld, nb) * cosP / l2;
                        mis = pL * pL / (pL * pL + pB * pB);
                    }
                    const V3 li = MatColor(S.mats[sl.mat]);
                    const V3 f = BxDF<ExactMath>(M, ray.d, ld, nb);
                    const float c = fabsf(Dot(ld, si.n));
                    lc = lc + mis * ray.T * (li * f * c * cosP / (pdfArea * l2));
                }
            }
        }
    } else if (S.envValid) {
        float r0, r1;
        s2.Next(r0, r1);
        float pdfuv = 0.0f;
        V3 li;
        const V3 sd = EnvSampleLit<ExactMath>(S, r0, r1, pdfuv, li);
        const V3 eo = si.pos + kEps * copysignf(1.0f, dt) * si.n;
        float d;
        if (TraverseWarp(S, eo, sd, 0.0f, kFltMax, d, stack, status) < 0) {
            const float c = fabsf(Dot(sd, si.n));
            const float sn = sqrtf(SMax(0.0f, 1.0f - c * c));
            const float pB = 2.0f * kPi * kPi * sn * BsdfPdf<ExactMath>(M, ray.d, sd, nb);
            const float mis = pdfuv * pdfuv / (pdfuv * pdfuv + pB * pB);
            const V3 f = BxDF<ExactMath>(M, ray.d, sd, nb);
            lc = lc + mis * ray.T * (li * f * sn * c * 2.0f * kPi * kPi) / pdfuv;
        }
    }
    return lc;
}

// PathTracing::Render (PathTracing.cpp:20-200)
__device__ void ReplayPtPixel(const DevScene& S, const DevCamera& C, const DevSettings& st, int px,
                              int py, float* film, RefSampler1D& s1, RefSampler2D& s2, const WarpStack& stack,
                              int* status) {
    V3 sum;
    for (int sp = 0; sp < st.spp; sp++) {
        V3 color;
        float r0, r1, r2, r3;
        s2.Next(r0, r1);
        s2.Next(r2, r3);
        Ray ray = GenerateRay<ExactMath>(C, px, py, st.width, st.height, r0, r1, r2, r3);
        Ray prev = ray;
        Shading si;
        {
            float d;
            const int k = TraverseWarp(S, ray.o, ray.d, 0.0f, kFltMax, d, stack, status);
            if (k < 0) {
                sum = sum + ray.T * EnvColor<ExactMath>(S, ray.d);
                continue;
            }
            si = Interpolate<ExactMath>(S, k, ray.o, ray.d, d);
        }
        if (IsEmission(S, si.mat)) {
            sum = sum + ray.T * MatColor(S.mats[si.mat]);
            continue;
        }
        for (int bounce = 0; bounce < st.maxBounces; bounce++) {
            DevMaterial Mh;
            const V3 nb = PointMaterial<ExactMath>(S, si.mat, si.slot, ray.o, ray.d, si.n, Mh);
            color = color + ReplayLight(S, si, Mh, nb, s1, s2, ray, stack, status);
            prev = ray;
            Shading sb = si;
            sb.n = nb;
            ray = NextRay<ExactMath>(Mh, ray, sb, s2);
            if (fabsf(SqLen(ray.T) - 0.0f) < kEps) break;
            float d;
            const int k = TraverseWarp(S, ray.o, ray.d, 0.0f, kFltMax, d, stack, status);
            if (k >= 0) {
                const Shading sn = Interpolate<ExactMath>(S, k, ray.o, ray.d, d);
                if (IsEmission(S, sn.mat)) {
                    const float l2 = SqLen(sn.pos - ray.o);
                    const float cosP = fabsf(Dot(ray.d, sn.n));
                    bool unused = false;
                    ReplaySampleLight(S, s1.Next(), s2, false, &unused);
                    const float pdfArea = S.lightPdfArea;
                    const float pB = BsdfPdf<ExactMath>(Mh, prev.d, ray.d, nb);
                    const float pL = l2 / cosP * pdfArea;
                    const float mis = pB * pB / (pL * pL + pB * pB);
                    color = color + mis * ray.T * MatColor(S.mats[sn.mat]);
                    break;
                }
                si = sn;
            } else {
                if (S.envValid) {
                    const float c = fabsf(Dot(si.n, ray.d));
                    const float sn = sqrtf(SMax(0.0f, 1.0f - c * c));
                    const float pB = BsdfPdf<ExactMath>(Mh, prev.d, ray.d, nb);
                    float mis = 0.0f;
                    if (ray.d.x != 0 && ray.d.y != 0 && sn > 0) {
                        const float pE = EnvPdf<ExactMath>(S, ray.d) / (2.0f * kPi * kPi * sn);
                        mis = pB * pB / (pE * pE + pB * pB);
                    } else {
                        mis = 1.0f;
                    }
                    color = color + mis * ray.T * EnvColor<ExactMath>(S, ray.d);
                } else {
                    color = color + ray.T * EnvColor<ExactMath>(S, ray.d);
                }
                break;
            }
        }
        if (MinElem(color) >= 0.0f) sum = sum + color;
    }
    const V3 avg = sum / (float)st.spp;
    if ((threadIdx.x & 31) == 0) {
        float* o = film + ((size_t)py * st.width + px) * 3;
        o[0] = avg.x;
        o[1] = avg.y;
        o[2] = avg.z;
    }
}

// One warp per tile of TileManager (Core/TileManager.cpp:8-43), every tile seeded
// RandomSampler1D(0) / RandomSampler2D(0, 1) as the Rendered pass does.
__global__ void __launch_bounds__(32) ReplayKernel(DevScene S, DevCamera C, DevSettings st,
                                                   float* __restrict__ film,
                                                   int* __restrict__ stackScratch,
                                                   int* __restrict__ statusOut, int tileBegin,
                                                   int tileEnd) {
    const int t = tileBegin + blockIdx.x;  // one warp per block, one tile per warp
    if (t >= tileEnd) return;
    const int nx = st.width / st.tileW, ny = st.height / st.tileH;
    const int remW = st.width - nx * st.tileW, remH = st.height - ny * st.tileH;
    const int ti = t % (nx + 1), tj = t / (nx + 1);
    if (tj > ny) return;
    const int x0 = ti * st.tileW, y0 = tj * st.tileH;
    const int w = (ti != nx) ? st.tileW : remW, h = (tj != ny) ? st.tileH : remH;
    __shared__ int4 sStack[kReplaySmemStack];
    const WarpStack stack{sStack, stackScratch + (size_t)(t - tileBegin) * S.stackDepth};
    int status = 0;
    RefSampler1D s1(0);
    RefSampler2D s2(0, 1);
    for (int y = y0; y < y0 + h; y++)
        for (int x = x0; x < x0 + w; x++) {
            if (st.integrator == kSimplePathTracing)
                ReplaySimplePixel(S, C, st, x, y, film, s1, s2, stack, &status);
            else
                ReplayPtPixel(S, C, st, x, y, film, s1, s2, stack, &status);
        }
    if (status && (threadIdx.x & 31) == 0) atomicOr(statusOut, status);
}

// ---------------------------------------------------------------- AOV passes
// Core/AOV/AOVUVCoordinate.cpp:11-51: numSamplesPerPixel camera rays, hit uvs summed.
__device__ void AovUVPixel(const DevScene& S, const DevCamera& C, const DevSettings& st, int px,
                           int py, float* film, RefSampler2D& s2, const WarpStack& stack, int* status) {
    V3 sum;
    for (int sp = 0; sp < st.spp; sp++) {
        float r0, r1, r2, r3;
        s2.Next(r0, r1);
        s2.Next(r2, r3);
        const Ray ray = GenerateRay<ExactMath>(C, px, py, st.width, st.height, r0, r1, r2, r3);
        float d;
        const int k = TraverseWarp(S, ray.o, ray.d, kEps, kInfinity, d, stack, status);
        if (k >= 0) sum = sum + InterpolateUV(S, k, ray.o, ray.d);
    }
    const V3 avg = sum / (float)st.spp;
    if ((threadIdx.x & 31) == 0) {
        float* o = film + ((size_t)py * st.width + px) * 3;
        o[0] = avg.x;
        o[1] = avg.y;
        o[2] = avg.z;
    }
}

// AOVDenoisingAlbedo.cpp:56-133 (normal == false), AOVDenoisingNormal.cpp:54-128 (normal ==
// true): glass and zero-roughness GGX are followed up to numMaxBounces; the first other
// surface, or the environment, gives the value. Emission gives zero (the reference's
// ASSERT(false) default branch in a release build).
__device__ V3 AovPath(const DevScene& S, const DevSettings& st, Ray ray, bool normal,
                      RefSampler1D& s1, RefSampler2D& s2, const WarpStack& stack, int* status) {
    for (int bounce = 0; bounce < st.maxBounces; bounce++) {
        float d;
        const int k = TraverseWarp(S, ray.o, ray.d, kEps, kInfinity, d, stack, status);
        if (k < 0) return normal ? ray.T * (-ray.d) : ray.T * EnvColor<ExactMath>(S, ray.d);
        const int m = ResolveMaterial(S.mats, SlotMaterial(S.shade, k), s1.Next());
        const Shading si = Interpolate<ExactMath>(S, k, ray.o, ray.d, d);
        DevMaterial M;
        Shading sb = si;
        sb.n = PointMaterial<ExactMath>(S, m, k, ray.o, ray.d, si.n, M);
        if (M.kind == kLambert) return normal ? ray.T * si.n : ray.T * V3(M.ar, M.ag, M.ab);
        if (M.kind == kGlossy && M.alpha != 0) return normal ? ray.T * si.n : ray.T * GgxF0(M);
        if (M.kind != kGlass && M.kind != kGlossy) return V3();
        ray = NextRay<ExactMath>(M, ray, sb, s2);  // Glass::GetAlpha is always 0
    }
    return V3();
}

__device__ void AovDenoisePixel(const DevScene& S, const DevCamera& C, const DevSettings& st,
                                bool normal, int dspp, int px, int py, float* film, RefSampler1D& s1,
                                RefSampler2D& s2, const WarpStack& stack, int* status) {
    V3 sum;
    for (int sp = 0; sp < dspp; sp++) {
        float r0, r1, r2, r3;
        s2.Next(r0, r1);
        s2.Next(r2, r3);
        const Ray ray = GenerateRay<ExactMath>(C, px, py, st.width, st.height, r0, r1, r2, r3);
        sum = sum + AovPath(S, st, ray, normal, s1, s2, stack, status);
    }
    const V3 avg = sum / (float)dspp;
    if ((threadIdx.x & 31) == 0) {
        float* o = film + ((size_t)py * st.width + px) * 3;
        o[0] = avg.x;
        o[1] = avg.y;
        o[2] = avg.z;
    }
}

// One warp per tile; unlike the Rendered pass, the AOV loops of Petrichor::Render
// (Core/Petrichor.cpp:104-261) advance tileIndex: tile k is seeded
// RandomSampler1D(k) / RandomSampler2D(k, k + 1).
__global__ void __launch_bounds__(32) AovKernel(DevScene S, DevCamera C, DevSettings st, int aov,
                                                int dspp, float* __restrict__ film,
                                                int* __restrict__ stackScratch,
                                                int* __restrict__ statusOut, int tileBegin,
                                                int tileEnd) {
    const int t = tileBegin + blockIdx.x;  // one warp per block, one tile per warp
    if (t >= tileEnd) return;
    const int nx = st.width / st.tileW, ny = st.height / st.tileH;
    const int remW = st.width - nx * st.tileW, remH = st.height - ny * st.tileH;
    const int ti = t % (nx + 1), tj = t / (nx + 1);
    if (tj > ny) return;
    const int x0 = ti * st.tileW, y0 = tj * st.tileH;
    const int w = (ti != nx) ? st.tileW : remW, h = (tj != ny) ? st.tileH : remH;
    __shared__ int4 sStack[kReplaySmemStack];
    const WarpStack stack{sStack, stackScratch + (size_t)(t - tileBegin) * S.stackDepth};
    int status = 0;
    RefSampler1D s1((uint32_t)t);
    RefSampler2D s2((uint32_t)t, (uint32_t)t + 1u);
    for (int y = y0; y < y0 + h; y++)
        for (int x = x0; x < x0 + w; x++) {
            if (aov == 0)
                AovUVPixel(S, C, st, x, y, film, s2, stack, &status);
            else
                AovDenoisePixel(S, C, st, aov == 2, dspp, x, y, film, s1, s2, stack, &status);
        }
    if (status && (threadIdx.x & 31) == 0) atomicOr(statusOut, status);
}

cudaError_t LaunchAov(const DevScene& S, const DevCamera& C, const DevSettings& st, int aov,
                      int dspp, float* film, int* stackScratch, int* status, int tileBegin,
                      int tileEnd, cudaStream_t stream) {
    const int n = tileEnd - tileBegin;
    if (n <= 0) return cudaSuccess;
    AovKernel<<<n, 32, 0, stream>>>(S, C, st, aov, dspp, film, stackScratch,
                                                              status, tileBegin, tileEnd);
    return cudaGetLastError();
}

__global__ void EnvTableExactKernel(DevScene S, float4* __restrict__ table) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < 2 * S.envH) EnvTableEntry<ExactMath>(S, e, table);
}
cudaError_t FillEnvTableExact(const DevScene& S, float4* table, cudaStream_t stream) {
    EnvTableExactKernel<<<(2 * S.envH + 31) / 32, 32, 0, stream>>>(S, table);
    return cudaGetLastError();
}

int NumTiles(const DevSettings& st) {
    return (st.width / st.tileW + 1) * (st.height / st.tileH + 1);
}

cudaError_t LaunchReplay(const DevScene& S, const DevCamera& C, const DevSettings& st, float* film,
                         int* stackScratch, int* status, int tileBegin, int tileEnd,
                         cudaStream_t stream) {
    const int n = tileEnd - tileBegin;
    if (n <= 0) return cudaSuccess;
    ReplayKernel<<<n, 32, 0, stream>>>(S, C, st, film, stackScratch,
                                                                 status, tileBegin, tileEnd);
    return cudaGetLastError();
}

}  // namespace ptg
