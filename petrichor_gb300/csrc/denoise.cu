// GPU denoiser in place of the reference's IntelOpenImageDenoiser
// (Core/Denoiser/IntelOpenImageDenoiser.cpp:15-101), which hands the film, and
// optionally the DenoisingAlbedo and DenoisingNormal AOVs, to Intel Open Image Denoise.
// That library and its trained weights are not part of this project, so the images
// differ from the reference's; the interface and the inputs are the same.
//
// Method: the edge-avoiding à-trous wavelet filter (H. Dammertz, D. Sewtz, J. Hanika,
// H. Lensch, "Edge-Avoiding À-Trous Wavelet Transform for fast Global Illumination
// Filtering", HPG 2010), with the luminance edge-stopping function scaled by a
// per-pixel noise estimate and that estimate carried through the iterations as in
// SVGF (C. Schied et al., HPG 2017):
//  - with an albedo, the colour is divided by it where it is not black (demodulation)
//    and multiplied back at the end, so texture detail is not blurred;
//  - the noise estimate is the variance of the (log, for HDR) luminance over a 3x3
//    window, blurred 3x3 before each pass;
//  - five passes of the 5x5 B3-spline kernel at steps 1, 2, 4, 8, 16 (clamped edges),
//    each tap weighted by exp(-|l_p - l_q| / (4 sigma_p)), (n_p . n_q)^128 where both
//    normals are known, and exp(-|a_p - a_q|^2 / 0.01) with an albedo; the centre tap
//    always has weight 1.
// Without AOVs the luminance stop is the only guide and is made stricter (2 sigma).
#include <cuda_runtime.h>

#include <cmath>
#include <utility>

#include "denoise.h"

namespace ptg {
namespace {

constexpr int kPasses = 5;
constexpr float kInvSigmaAlbedo2 = 1.0f / (0.1f * 0.1f);

__device__ __forceinline__ float Lum(float r, float g, float b) {
    return 0.2126f * r + 0.7152f * g + 0.0722f * b;
}
__device__ __forceinline__ float EdgeLum(float r, float g, float b, int hdr) {
    const float y = fmaxf(Lum(r, g, b), 0.0f);
    return hdr ? log1pf(y) : fminf(y, 1.0f);
}
__device__ __forceinline__ int Clamp(int v, int hi) { return v < 0 ? 0 : (v > hi ? hi : v); }

// 2^x (relative error 2^-22; results below 2^-126 are 0)
__device__ __forceinline__ float Exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct Planes {
    int W, H, hdr;
    float4* color;   // demodulated colour .xyz, edge luminance .w (two buffers)
    float4* color2;
    float* var;      // per-pixel luminance variance (two buffers)
    float* var2;
    float4* albedo;  // demodulation factor .xyz, 1 where the albedo guide applies (with an albedo)
    float4* normal;  // normal .xyz of length sqrt(1/2), 1 where known (with a normal)
};

// One pixel's demodulated colour, demodulation factor and edge luminance.
__device__ __forceinline__ float4 Demodulate(const float* __restrict__ color, const float* __restrict__ albedo,
                                             size_t p, int hdr, float4& a) {
    float r = color[3 * p], g = color[3 * p + 1], b = color[3 * p + 2];
    if (!isfinite(r) || !isfinite(g) || !isfinite(b)) r = g = b = 0.0f;
    a = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    if (albedo) {
        const float ar = albedo[3 * p], ag = albedo[3 * p + 1], ab = albedo[3 * p + 2];
        a.w = 1.0f;  // the albedo edge stop applies
        if (isfinite(ar) && isfinite(ag) && isfinite(ab) && Lum(ar, ag, ab) > 0.01f) {
            a.x = fmaxf(ar, 1e-3f);
            a.y = fmaxf(ag, 1e-3f);
            a.z = fmaxf(ab, 1e-3f);
        }
        if (!(isfinite(ar) && isfinite(ag) && isfinite(ab))) a.w = 0.0f;
        r /= a.x;
        g /= a.y;
        b /= a.z;
    }  // the albedo edge stop compares these factors (the albedo, or 1 where it is black)
    return make_float4(r, g, b, EdgeLum(r, g, b, hdr));
}

// Demodulated colours, guides and the 3x3 variance of the edge luminance. A block covers
// kPrepW x kPrepH pixels; the luminances of its tile and the pixels around it are formed
// in shared memory (1.3 times the pixels), which spares a second pass over the image.
constexpr int kPrepW = 32, kPrepH = 8;
__global__ void __launch_bounds__(kPrepW* kPrepH) PrepKernel(Planes P, const float* __restrict__ color,
                                                            const float* __restrict__ albedo,
                                                            const float* __restrict__ normal) {
    __shared__ float lum[kPrepH + 2][kPrepW + 2];
    const int x0 = blockIdx.x * kPrepW, y0 = blockIdx.y * kPrepH;
    for (int i = threadIdx.x; i < (kPrepW + 2) * (kPrepH + 2); i += kPrepW * kPrepH) {
        const int tx = i % (kPrepW + 2), ty = i / (kPrepW + 2);
        const int x = Clamp(x0 + tx - 1, P.W - 1), y = Clamp(y0 + ty - 1, P.H - 1);
        const size_t p = (size_t)y * P.W + x;
        float4 a;
        const float4 c = Demodulate(color, albedo, p, P.hdr, a);
        lum[ty][tx] = c.w;
        if (tx >= 1 && tx <= kPrepW && ty >= 1 && ty <= kPrepH && x == x0 + tx - 1 && y == y0 + ty - 1) {
            P.color[p] = c;
            if (albedo) P.albedo[p] = a;
        }
    }
    __syncthreads();
    const int tx = threadIdx.x % kPrepW, ty = threadIdx.x / kPrepW;
    const int x = x0 + tx, y = y0 + ty;
    if (x >= P.W || y >= P.H) return;
    const size_t p = (size_t)y * P.W + x;
    if (normal) {
        float4 n = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float nx = normal[3 * p], ny = normal[3 * p + 1], nz = normal[3 * p + 2];
        const float l2 = fmaf(nx, nx, fmaf(ny, ny, nz * nz));
        if (isfinite(l2) && l2 > 0.25f) {
            const float inv = 0.70710678f / sqrtf(l2);
            n = make_float4(nx * inv, ny * inv, nz * inv, 1.0f);
        }
        P.normal[p] = n;
    }
    float m1 = 0.0f, m2 = 0.0f;
    for (int dy = 0; dy < 3; dy++)
        for (int dx = 0; dx < 3; dx++) {
            const float l = lum[ty + dy][tx + dx];
            m1 += l;
            m2 += l * l;
        }
    m1 *= 1.0f / 9.0f;
    m2 *= 1.0f / 9.0f;
    P.var[p] = fmaxf(m2 - m1 * m1, 0.0f);
}

// One a-trous pass. A thread filters kRows pixels of one column, `step` rows apart, whose 5x5
// windows share their taps: kRows + 4 rows of 5 taps are loaded for kRows pixels (12 taps
// a pixel instead of 25). A warp's lanes are 32 neighbouring columns, so every load is a
// run of whole sectors whatever the step. Bound by issue (70-76% of the slots, about 33
// instructions a tap and pixel): the luminance and albedo stops share one exponential, and
// the normal stop's 128th power is seven squarings (more exact than a logarithm and a
// power, and faster: the exponential unit is the next limit).
// The 3x3 blur of the variance (at the pass's own pixel) and, in the last pass, the
// multiplication by the albedo factor are formed here too.
// 1920x1080 with both guides: 874 us in 13 launches with one pixel a thread, 474 us in 6.
// Rows x blocks per SM (before the normal stop's difference form): 3x4 498, 2x6 517, 3x5 554,
// 2x4 562, 4x4 597, 1x8 682 us.
constexpr int kRows = 3;
template <bool kNormal, bool kAlbedo>
__global__ void __launch_bounds__(128, 4) ATrousKernel(Planes P, int step, float sigmaLum, float* __restrict__ out) {
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    // group g: rows y0 + step * j of the band of kRows * step rows it lies in
    const int g = blockIdx.y * 4 + (threadIdx.x >> 5);
    const int y0 = g / step * (kRows * step) + g % step;
    if (x >= P.W || y0 >= P.H) return;
    constexpr float kLog2e = 1.44269504f;
    float4 ap[kRows], np[kRows];
    float lp[kRows], scale[kRows];
    float sr[kRows], sg[kRows], sb[kRows], sw[kRows], sv[kRows];
#pragma unroll
    for (int j = 0; j < kRows; j++) {
        const int y = min(y0 + j * step, P.H - 1);
        const size_t p = (size_t)y * P.W + x;
        float s = 0.0f;
        for (int dy = -1; dy <= 1; dy++) {
            const float* row = P.var + (size_t)Clamp(y + dy, P.H - 1) * P.W;
            s += row[Clamp(x - 1, P.W - 1)] + row[x] + row[Clamp(x + 1, P.W - 1)];
        }
        // log2(e) folded in: the stops are powers of two
        scale[j] = kLog2e / (sigmaLum * sqrtf(s * (1.0f / 9.0f)) + 1e-4f);
        lp[j] = P.color[p].w;
        if (kAlbedo) ap[j] = P.albedo[p];
        if (kNormal) np[j] = P.normal[p];
        sr[j] = sg[j] = sb[j] = sw[j] = sv[j] = 0.0f;
    }
    const float h[5] = {1.0f / 16.0f, 1.0f / 4.0f, 3.0f / 8.0f, 1.0f / 4.0f, 1.0f / 16.0f};
#pragma unroll 1
    for (int kx = 0; kx < 5; kx++) {
        const int qx = Clamp(x + (kx - 2) * step, P.W - 1);
        const float hx = kx == 2 ? 3.0f / 8.0f : (kx == 1 || kx == 3) ? 1.0f / 4.0f : 1.0f / 16.0f;
#pragma unroll
        for (int t = 0; t < kRows + 4; t++) {
            const size_t q = (size_t)Clamp(y0 + (t - 2) * step, P.H - 1) * P.W + qx;
            const float4 cq = P.color[q];
            const float vq = P.var[q];
            float4 aq, nq;
            if (kAlbedo) aq = P.albedo[q];
            if (kNormal) nq = P.normal[q];
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int ky = t - j;
                if (ky < 0 || ky > 4) continue;
                float e = -fabsf(lp[j] - cq.w) * scale[j];
                if (kAlbedo) {
                    const float dr = ap[j].x - aq.x, dg = ap[j].y - aq.y, db = ap[j].z - aq.z;
                    const float d2 = fmaf(dr, dr, fmaf(dg, dg, db * db));
                    if (ap[j].w > 0.0f && aq.w > 0.0f) e = fmaf(d2, -kInvSigmaAlbedo2 * kLog2e, e);
                }
                float w = Exp2(e);
                if (kNormal) {
                    // the cosine as 1 - |n_p - n_q|^2 / 2: exactly 1 for equal normals, where the
                    // 128th power would raise the rounding of a dot product
                    const float nx = np[j].x - nq.x, ny = np[j].y - nq.y, nz = np[j].z - nq.z;
                    float d = fmaxf(0.0f, fmaf(-nx, nx, fmaf(-ny, ny, fmaf(-nz, nz, 1.0f))));
#pragma unroll
                    for (int k = 0; k < 7; k++) d *= d;  // d^128
                    if (np[j].w > 0.0f && nq.w > 0.0f) w *= d;
                }
                if (ky == 2 && kx == 2) w = 1.0f;  // the centre tap
                const float wh = w * (h[ky] * hx);
                sr[j] = fmaf(wh, cq.x, sr[j]);
                sg[j] = fmaf(wh, cq.y, sg[j]);
                sb[j] = fmaf(wh, cq.z, sb[j]);
                sw[j] += wh;
                sv[j] = fmaf(wh * wh, vq, sv[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kRows; j++) {
        const int y = y0 + j * step;
        if (y >= P.H) break;
        const size_t p = (size_t)y * P.W + x;
        const float inv = 1.0f / sw[j];  // sw >= h2 * h2 > 0 (centre tap)
        float r = sr[j] * inv, g2 = sg[j] * inv, b = sb[j] * inv;
        if (out) {
            if (kAlbedo) {
                r *= ap[j].x;
                g2 *= ap[j].y;
                b *= ap[j].z;
            }
            out[3 * p] = r;
            out[3 * p + 1] = g2;
            out[3 * p + 2] = b;
        } else {
            P.color2[p] = make_float4(r, g2, b, EdgeLum(r, g2, b, P.hdr));
            P.var2[p] = sv[j] * inv * inv;
        }
    }
}

using ATrous = void (*)(Planes, int, float, float*);
ATrous Pass(bool normal, bool albedo) {
    return normal ? (albedo ? ATrousKernel<true, true> : ATrousKernel<true, false>)
                  : (albedo ? ATrousKernel<false, true> : ATrousKernel<false, false>);
}

}  // namespace

size_t DenoiseScratchBytes(int width, int height) {
    const size_t n = (size_t)width * height;
    return n * (4 * sizeof(float4) + 2 * sizeof(float)) + 6 * 256;  // 6 planes, 256-aligned
}

cudaError_t Denoise(int width, int height, const float* color, const float* albedo,
                    const float* normal, int hdr, float* out, void* scratch, cudaStream_t stream,
                    int* launches) {
    const size_t n = (size_t)width * height;
    char* s = static_cast<char*>(scratch);
    auto carve = [&](size_t bytes) {
        char* p = s;
        s += (bytes + 255) / 256 * 256;
        return p;
    };
    Planes P;
    P.W = width;
    P.H = height;
    P.hdr = hdr ? 1 : 0;
    P.color = reinterpret_cast<float4*>(carve(n * sizeof(float4)));
    P.color2 = reinterpret_cast<float4*>(carve(n * sizeof(float4)));
    P.albedo = reinterpret_cast<float4*>(carve(n * sizeof(float4)));
    P.normal = reinterpret_cast<float4*>(carve(n * sizeof(float4)));
    P.var = reinterpret_cast<float*>(carve(n * sizeof(float)));
    P.var2 = reinterpret_cast<float*>(carve(n * sizeof(float)));
    const float sigmaLum = (albedo || normal) ? 4.0f : 2.0f;
    PrepKernel<<<dim3((width + kPrepW - 1) / kPrepW, (height + kPrepH - 1) / kPrepH), kPrepW * kPrepH, 0, stream>>>(
      P, color, albedo, normal);
    const ATrous filter = Pass(normal != nullptr, albedo != nullptr);
    for (int pass = 0; pass < kPasses; pass++) {
        const int step = 1 << pass;
        const int groups = (height + kRows * step - 1) / (kRows * step) * step;
        filter<<<dim3((width + 31) / 32, (groups + 3) / 4), 128, 0, stream>>>(
          P, step, sigmaLum, pass == kPasses - 1 ? out : nullptr);
        std::swap(P.color, P.color2);
        std::swap(P.var, P.var2);
    }
    const int k = 1 + kPasses;
    if (launches) *launches += k;
    return cudaGetLastError();
}

}  // namespace ptg
