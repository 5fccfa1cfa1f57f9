// Post-process (postprocess.glsl:26-171 with TiledRenderer's uniforms, TiledRenderer.cpp:540-552):
// mean of the accumulated radiance (optionally with chromatic aberration), one of the seven
// tone maps with the shader's gamma, optional vignette, then the 8-bit framebuffer conversion
// (clamp to [0, 1], round to nearest) that GetOutputBuffer reads back. The accumulation buffer
// is sampled as the shader's GL_LINEAR / GL_REPEAT texture, with the filtering contract of the
// environment map (texel centres at +0.5, float weights).
#define LF_CONTRACT_INLINE   // three independent channels of pow: inline they overlap
#include "lf_internal.h"

#include <algorithm>

#include "../lf_contract.h"

namespace lfd
{
namespace
{
struct PostParams
{
    int tonemap;
    int useCA, useCADistortion, useVignette, preview;
    float caDistance, caP1, caP2, caP3, vignetteIntensity, vignettePower;
    float invSamples;
};

__device__ __forceinline__ int wrapi(int i, int n)
{
    if ((unsigned)i < (unsigned)n) return i;
    int r = i % n;
    return r < 0 ? r + n : r;
}

// texture(pathTraceTexture, uv): bilinear, GL_REPEAT, channel c of the RGB sums.
__device__ __forceinline__ float tex_bilinear(const float4* t, int w, int h, float u, float v, int c)
{
    const float xf = u * (float)w - 0.5f, yf = v * (float)h - 0.5f;
    const float fx0 = floorf(xf), fy0 = floorf(yf);
    const float a = xf - fx0, b = yf - fy0;
    const int x0 = wrapi((int)fx0, w), x1 = wrapi((int)fx0 + 1, w);
    const int y0 = wrapi((int)fy0, h), y1 = wrapi((int)fy0 + 1, h);
    auto at = [&](int x, int y) {
        const float4 p = t[(size_t)y * w + x];
        return c == 0 ? p.x : (c == 1 ? p.y : p.z);
    };
    const float ia = 1.0f - a, ib = 1.0f - b;
    const float top = at(x0, y0) * ia + at(x1, y0) * a;
    const float bot = at(x0, y1) * ia + at(x1, y1) * a;
    return top * ib + bot * b;
}

__device__ __forceinline__ float distance2(float ax, float ay, float bx, float by)
{
    const float dx = ax - bx, dy = ay - by;
    return sqrtf(dx * dx + dy * dy);
}

__device__ __forceinline__ float clamp01(float x) { return lfc::clamp_g(x, 0.0f, 1.0f); }

// Tone map `idx` of the three colour channels (the shader's alpha is not read back).
__device__ void tonemap(int idx, float c[3])
{
    const float g = 1.0f / 2.2f;
    if (idx == 1)
    {
        // tonemap(c, 2): c * 1.0 / (1.0 + luminance / limit)
        const float lum = 0.3f * c[0] + 0.6f * c[1] + 0.1f * c[2];
        const float den = 1.0f + lum / 2.0f;
        for (int k = 0; k < 3; ++k) c[k] = lfc::pow_c(c[k] * 1.0f / den, g);
    }
    else if (idx == 2)
    {
        const float a = 2.51f, b = 0.03f, y = 2.43f, d = 0.59f, e = 0.14f;
        for (int k = 0; k < 3; ++k)
            c[k] = lfc::pow_c(clamp01((c[k] * (a * c[k] + b)) / (c[k] * (y * c[k] + d) + e)), g);
    }
    else if (idx == 3)
    {
        for (int k = 0; k < 3; ++k) c[k] = lfc::pow_c(clamp01(c[k] / (c[k] + 1.0f)), g);
    }
    else if (idx == 4)
    {
        const float a = 1.2295f, b = 0.3135f, y = 1.1935f, d = 0.4655f, e = 0.073f;
        for (int k = 0; k < 3; ++k)
        {
            float v = lfc::pow_c((c[k] * (c[k] * (a * c[k] + b) + y * d) / (c[k] * (y * c[k] + d) + e)), 1.7f);
            v = lfc::pow_c(v, 1.0f / 0.8f);
            v = v * 0.8f;
            c[k] = lfc::pow_c(clamp01(v), g);
        }
    }
    else if (idx == 5)
    {
        for (int k = 0; k < 3; ++k)
        {
            const float v = lfc::fmax_g(0.0f, c[k] - 0.004f);
            c[k] = (v * (6.2f * v + 0.5f)) / (v * (6.2f * v + 1.7f) + 0.06f);
        }
    }
    else if (idx == 6)
    {
        const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, E = 0.02f, F = 0.30f;
        for (int k = 0; k < 3; ++k)
        {
            const float v = ((c[k] * (A * c[k] + C * B) + D * E) / (c[k] * (A * c[k] + B) + D * F)) - E / F;
            c[k] = lfc::pow_c(v, g) * 1.75f;
        }
    }
}
}

// One thread per pixel; a block's 256 pixels are packed in shared memory and written as 4-byte and
// 16-byte words, in the caller's layout (3 bytes and 3 floats a pixel): on a coherent host into the
// caller's buffers, else into device buffers that are copied there. With padded pixels, copied into
// temporaries and repacked by the host, 1920 x 1080 took 4.0 ms; over copies 0.27 ms, of which the
// kernel is 77 us (pow, bound by instruction issue; 95 us with the transcendental functions out of
// line) and most of the rest the copies at 180 GB/s; written directly 0.21 ms (31 MB over C2C beside
// the arithmetic). Copies to pageable memory wait for the stream, so splitting the image
// into bands to overlap them only adds waits (two bands 317 us against 296, four 368).
constexpr int kPostBlock = 256;

__global__ void __launch_bounds__(kPostBlock) postprocess_kernel(const float4* accum, int W, int H, PostParams P,
                                                                 uint8_t* out8, float* outf)
{
    __shared__ __align__(16) float sf[3 * kPostBlock];
    __shared__ __align__(16) uint8_t s8[3 * kPostBlock];
    const int t = threadIdx.x, n = W * H;
    for (int base = blockIdx.x * kPostBlock; base < n; base += gridDim.x * kPostBlock)
    {
        const int i = base + t;
        if (i < n)
        {
            const int x = i % W, y = i / W;
            const float u = ((float)x + 0.5f) / (float)W, v = ((float)y + 0.5f) / (float)H;
            float c[3];
            if (!P.preview && P.useCA)
            {
                float offset = P.caDistance;
                const float dist = 0.0f + lfc::pow_c(distance2(u, v, P.caP3, P.caP3), P.caP1) * P.caP2;
                float su, sv;
                if (P.useCADistortion)
                    su = sv = offset * dist;
                else
                {
                    offset = offset * 0.025f;
                    su = sv = offset * P.caP2;
                }
                c[0] = tex_bilinear(accum, W, H, u + su, v + sv, 0) * P.invSamples;
                c[1] = tex_bilinear(accum, W, H, u, v, 1) * P.invSamples;
                c[2] = tex_bilinear(accum, W, H, u - su, v - sv, 2) * P.invSamples;
            }
            else
                for (int k = 0; k < 3; ++k) c[k] = tex_bilinear(accum, W, H, u, v, k) * P.invSamples;
            tonemap(P.tonemap, c);
            if (P.useVignette)
            {
                const float dist = 1.0f - lfc::pow_c(distance2(u, v, 0.5f, 0.5f), P.vignettePower) * P.vignetteIntensity;
                for (int k = 0; k < 3; ++k) c[k] = c[k] * dist;
            }
            for (int k = 0; k < 3; ++k)
            {
                sf[3 * t + k] = c[k];
                s8[3 * t + k] = (uint8_t)rintf(clamp01(c[k]) * 255.0f);
            }
        }
        __syncthreads();
        const int m = 3 * (n - base < kPostBlock ? n - base : kPostBlock);   // values of this block
        if (outf)
        {
            float* dst = outf + (size_t)3 * base;
            for (int k = 4 * t; k + 3 < m; k += 4 * kPostBlock)
                *reinterpret_cast<float4*>(dst + k) = *reinterpret_cast<const float4*>(sf + k);
            for (int k = (m & ~3) + t; k < m; k += kPostBlock) dst[k] = sf[k];
        }
        if (out8)
        {
            uint8_t* dst = out8 + (size_t)3 * base;
            for (int k = 4 * t; k + 3 < m; k += 4 * kPostBlock)
                *reinterpret_cast<uint32_t*>(dst + k) = *reinterpret_cast<const uint32_t*>(s8 + k);
            for (int k = (m & ~3) + t; k < m; k += kPostBlock) dst[k] = s8[k];
        }
        __syncthreads();
    }
}
}

using namespace lfrt;

extern "C" lf_status lf_frame_postprocess(lf_frame* f, const lf_post_params* pp, int32_t samples, uint8_t* rgb8,
                                          float* rgbf)
{
    if (!f || !pp || samples <= 0 || (!rgb8 && !rgbf) || pp->tonemap < 0 || pp->tonemap > 6) return LF_ERR_INVALID;
    lf_ctx* c = f->ctx;
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    cudaSetDevice(c->device);
    const size_t pix = (size_t)f->W * f->H;
    // results go straight to the caller's buffers where the kernel can write there, else over device
    // buffers
    const bool direct8 = rgb8 && direct_host(c, rgb8, pix * 3, true, 4);
    const bool directf = rgbf && direct_host(c, rgbf, pix * 3 * sizeof(float), true);
    uint8_t* d8 = direct8 ? rgb8 : nullptr;
    float* df = directf ? rgbf : nullptr;
    cudaError_t e = cudaSuccess;
    if (rgb8 && !direct8) e = pool_alloc(c, &d8, pix * 3, c->stream);
    if (e == cudaSuccess && rgbf && !directf) e = pool_alloc(c, &df, pix * 3 * sizeof(float), c->stream);
    if (e != cudaSuccess)
    {
        if (d8 && !direct8) cudaFreeAsync(d8, c->stream);
        return cuda_fail(c, e, "post-process buffers");
    }
    PostParams P;
    P.tonemap = pp->tonemap;
    P.useCA = pp->use_ca;
    P.useCADistortion = pp->use_ca_distortion;
    P.useVignette = pp->use_vignette;
    P.preview = pp->preview;
    P.caDistance = pp->ca_distance;
    P.caP1 = pp->ca_p1;
    P.caP2 = pp->ca_p2;
    P.caP3 = pp->ca_p3;
    P.vignetteIntensity = pp->vignette_intensity;
    P.vignettePower = pp->vignette_power;
    P.invSamples = 1.0f / (float)samples;
    const int grid = (int)std::min<size_t>((pix + kPostBlock - 1) / kPostBlock, 152 * 16);
    postprocess_kernel<<<grid, kPostBlock, 0, c->stream>>>(f->accum, f->W, f->H, P, d8, df);
    e = cudaGetLastError();
    if (rgb8 && !direct8)
    {
        if (e == cudaSuccess) e = cudaMemcpyAsync(rgb8, d8, pix * 3, cudaMemcpyDeviceToHost, c->stream);
        cudaFreeAsync(d8, c->stream);
    }
    if (rgbf && !directf)
    {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(rgbf, df, pix * 3 * sizeof(float), cudaMemcpyDeviceToHost, c->stream);
        cudaFreeAsync(df, c->stream);
    }
    const lf_status st = check_device(c);
    return e == cudaSuccess ? st : cuda_fail(c, e, "post-process");
}
