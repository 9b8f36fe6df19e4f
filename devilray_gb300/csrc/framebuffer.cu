// framebuffer.cu -- accumulation buffers of a progressive render and their
// display conversion on the device (Renderer::createPixels of the reference,
// src/Renderer.cpp:51-90, which copies the whole buffer to the host each frame).

#include "dr_internal.h"
#include "alias_kernels.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

struct dr_framebuffer {
    dr_context *ctx = nullptr;
    int32_t width = 0, height = 0;
    float4 *accum = nullptr;
    uint32_t *casts = nullptr;
    uint32_t *pixels = nullptr;
};

namespace dr {
namespace {

__device__ __forceinline__ uint32_t to_u32(float f) { return (uint32_t)roundf(f); }

// The sRGB byte of createPixels: with r the value clamped to [0, 1], round(255 s),
// s = 12.92 r below 0.0031308, else 1.055 r^(1/2.4) - 0.055, in the
// reference's mix of types: a correctly rounded FP32 power, the rest of the
// expression in double, s and 255 s rounded to FP32. kSrgbStep[n] is the
// smallest FP32 r whose byte is above n, found by bisection over that
// expression (which is monotonic around every step).
__constant__ float kSrgbStep[255] = {
    0x1.3e4568p-13f, 0x1.dd681cp-12f, 0x1.8dd6c2p-11f, 0x1.167cbcp-10f, 0x1.660e16p-10f, 0x1.b59f6ep-10f,
    0x1.029864p-9f, 0x1.2a6112p-9f, 0x1.5229bep-9f, 0x1.79f26cp-9f, 0x1.a1e59cp-9f, 0x1.cbf72ep-9f,
    0x1.f86802p-9f, 0x1.13a0bcp-8f, 0x1.2c4662p-8f, 0x1.462978p-8f, 0x1.614e5ep-8f, 0x1.7db96ap-8f,
    0x1.9b6ed8p-8f, 0x1.ba72ccp-8f, 0x1.dac95cp-8f, 0x1.fc7688p-8f, 0x1.0fbf20p-7f, 0x1.21f232p-7f,
    0x1.34d660p-7f, 0x1.486d8ap-7f, 0x1.5cb98ep-7f, 0x1.71bc32p-7f, 0x1.877746p-7f, 0x1.9dec8cp-7f,
    0x1.b51dc4p-7f, 0x1.cd0ca2p-7f, 0x1.e5bae0p-7f, 0x1.ff2a1cp-7f, 0x1.0cae02p-6f, 0x1.1a291cp-6f,
    0x1.280728p-6f, 0x1.3648f4p-6f, 0x1.44ef48p-6f, 0x1.53faeep-6f, 0x1.636ca4p-6f, 0x1.73452ep-6f,
    0x1.83854ep-6f, 0x1.942dc2p-6f, 0x1.a53f44p-6f, 0x1.b6ba90p-6f, 0x1.c8a05ep-6f, 0x1.daf168p-6f,
    0x1.edae5ap-6f, 0x1.006bf6p-5f, 0x1.0a3766p-5f, 0x1.1439d6p-5f, 0x1.1e739ep-5f, 0x1.28e510p-5f,
    0x1.338e8ap-5f, 0x1.3e7056p-5f, 0x1.498acep-5f, 0x1.54de42p-5f, 0x1.606b06p-5f, 0x1.6c316cp-5f,
    0x1.7831c4p-5f, 0x1.846c60p-5f, 0x1.90e190p-5f, 0x1.9d91a0p-5f, 0x1.aa7ce0p-5f, 0x1.b7a3a0p-5f,
    0x1.c50632p-5f, 0x1.d2a4d4p-5f, 0x1.e07fdcp-5f, 0x1.ee9794p-5f, 0x1.fcec46p-5f, 0x1.05bf20p-4f,
    0x1.0d26e4p-4f, 0x1.14ad94p-4f, 0x1.1c5354p-4f, 0x1.24184cp-4f, 0x1.2bfc9ap-4f, 0x1.340068p-4f,
    0x1.3c23d4p-4f, 0x1.446704p-4f, 0x1.4cca1cp-4f, 0x1.554d40p-4f, 0x1.5df08ep-4f, 0x1.66b42ap-4f,
    0x1.6f9836p-4f, 0x1.789cd4p-4f, 0x1.81c226p-4f, 0x1.8b0850p-4f, 0x1.946f70p-4f, 0x1.9df7a8p-4f,
    0x1.a7a11ap-4f, 0x1.b16be6p-4f, 0x1.bb582ep-4f, 0x1.c56610p-4f, 0x1.cf95acp-4f, 0x1.d9e726p-4f,
    0x1.e45a9ep-4f, 0x1.eef02ep-4f, 0x1.f9a7f6p-4f, 0x1.02410ep-3f, 0x1.07bf5cp-3f, 0x1.0d4ef6p-3f,
    0x1.12efeap-3f, 0x1.18a24cp-3f, 0x1.1e6626p-3f, 0x1.243b88p-3f, 0x1.2a2284p-3f, 0x1.301b28p-3f,
    0x1.362580p-3f, 0x1.3c41a0p-3f, 0x1.426f92p-3f, 0x1.48af6ap-3f, 0x1.4f0132p-3f, 0x1.5564f8p-3f,
    0x1.5bdacep-3f, 0x1.6262c0p-3f, 0x1.68fcdep-3f, 0x1.6fa936p-3f, 0x1.7667d6p-3f, 0x1.7d38ccp-3f,
    0x1.841c28p-3f, 0x1.8b11f4p-3f, 0x1.921a42p-3f, 0x1.99351ep-3f, 0x1.a06296p-3f, 0x1.a7a2b8p-3f,
    0x1.aef592p-3f, 0x1.b65b32p-3f, 0x1.bdd3a4p-3f, 0x1.c55ef8p-3f, 0x1.ccfd3ap-3f, 0x1.d4ae78p-3f,
    0x1.dc72bep-3f, 0x1.e44a1cp-3f, 0x1.ec349ep-3f, 0x1.f43252p-3f, 0x1.fc4342p-3f, 0x1.0233c0p-2f,
    0x1.064f8cp-2f, 0x1.0a7508p-2f, 0x1.0ea440p-2f, 0x1.12dd36p-2f, 0x1.171ff4p-2f, 0x1.1b6c7ep-2f,
    0x1.1fc2dap-2f, 0x1.242312p-2f, 0x1.288d28p-2f, 0x1.2d0124p-2f, 0x1.317f12p-2f, 0x1.3606eep-2f,
    0x1.3a98c2p-2f, 0x1.3f3496p-2f, 0x1.43da70p-2f, 0x1.488a54p-2f, 0x1.4d444ap-2f, 0x1.52085ap-2f,
    0x1.56d686p-2f, 0x1.5baed6p-2f, 0x1.609152p-2f, 0x1.657dfep-2f, 0x1.6a74e0p-2f, 0x1.6f75fep-2f,
    0x1.74815ep-2f, 0x1.799706p-2f, 0x1.7eb6fep-2f, 0x1.83e148p-2f, 0x1.8915eep-2f, 0x1.8e54f4p-2f,
    0x1.939e5ep-2f, 0x1.98f236p-2f, 0x1.9e507ep-2f, 0x1.a3b93ep-2f, 0x1.a92c7cp-2f, 0x1.aeaa3cp-2f,
    0x1.b43284p-2f, 0x1.b9c55cp-2f, 0x1.bf62c8p-2f, 0x1.c50acep-2f, 0x1.cabd78p-2f, 0x1.d07ac4p-2f,
    0x1.d642b8p-2f, 0x1.dc155ep-2f, 0x1.e1f2bap-2f, 0x1.e7dad2p-2f, 0x1.edcdacp-2f, 0x1.f3cb4cp-2f,
    0x1.f9d3bap-2f, 0x1.ffe6f8p-2f, 0x1.030288p-1f, 0x1.061702p-1f, 0x1.0930ecp-1f, 0x1.0c504cp-1f,
    0x1.0f7520p-1f, 0x1.129f70p-1f, 0x1.15cf3cp-1f, 0x1.190486p-1f, 0x1.1c3f52p-1f, 0x1.1f7fa2p-1f,
    0x1.22c578p-1f, 0x1.2610d8p-1f, 0x1.2961c6p-1f, 0x1.2cb840p-1f, 0x1.30144ep-1f, 0x1.3375f0p-1f,
    0x1.36dd28p-1f, 0x1.3a49f8p-1f, 0x1.3dbc66p-1f, 0x1.413474p-1f, 0x1.44b224p-1f, 0x1.483576p-1f,
    0x1.4bbe6ep-1f, 0x1.4f4d10p-1f, 0x1.52e15cp-1f, 0x1.567b58p-1f, 0x1.5a1b04p-1f, 0x1.5dc062p-1f,
    0x1.616b78p-1f, 0x1.651c46p-1f, 0x1.68d2cep-1f, 0x1.6c8f14p-1f, 0x1.70511ap-1f, 0x1.7418e2p-1f,
    0x1.77e670p-1f, 0x1.7bb9c6p-1f, 0x1.7f92e6p-1f, 0x1.8371d2p-1f, 0x1.87568cp-1f, 0x1.8b4118p-1f,
    0x1.8f317ap-1f, 0x1.9327b0p-1f, 0x1.9723c0p-1f, 0x1.9b25acp-1f, 0x1.9f2d76p-1f, 0x1.a33b1ep-1f,
    0x1.a74eaap-1f, 0x1.ab681cp-1f, 0x1.af8776p-1f, 0x1.b3acb8p-1f, 0x1.b7d7ecp-1f, 0x1.bc090ap-1f,
    0x1.c0401ap-1f, 0x1.c47d1cp-1f, 0x1.c8c016p-1f, 0x1.cd0908p-1f, 0x1.d157f4p-1f, 0x1.d5acdep-1f,
    0x1.da07c6p-1f, 0x1.de68b2p-1f, 0x1.e2cfa0p-1f, 0x1.e73c96p-1f, 0x1.ebaf94p-1f, 0x1.f0289ep-1f,
    0x1.f4a7b6p-1f, 0x1.f92cdep-1f, 0x1.fdb818p-1f};

// FP32 with the hardware logarithm and exponential gives 255 s to within 4e-4
// (log2: 2^-22 x 8.4 over [0.0031, 1]; exp2: 2 ulp; the roundings of the
// product and of the sum), so the byte is certain unless 255 s lies within
// kSrgbDoubt of a rounding boundary n + 1/2 (0.2 % of values); there the exact
// step decides. The double power that this replaces ran at 1/64 of the FP32
// rate and bound the whole conversion: 1080p 1,036 us with it, 18.4 us without
// (equal bytes for every FP32 value in [0, 1]).
constexpr float kSrgbDoubt = 1e-3f;
// The byte of the channel sum / samples, inv within an ulp of 1 / samples: the
// estimate takes the product, the steps the quotient itself.
__device__ __forceinline__ uint32_t srgb_byte(float sum, float samples, float inv)
{
    const float r = fminf(fmaxf(sum * inv, 0.f), 1.f);
    const float v = r < 0.0031308f ? r * (12.92f * 255.0f)
                                   : exp2f(__log2f(r) * (1 / 2.4f)) * (1.055f * 255.0f) - 0.055f * 255.0f;
    const float n = floorf(v);
    if (fabsf(v - n - 0.5f) < kSrgbDoubt) {
        const float q = fminf(fmaxf(sum / samples, 0.f), 1.f);
        return (uint32_t)n + (q >= kSrgbStep[(int)n] ? 1u : 0u);
    }
    return (uint32_t)(v + 0.5f);
}

__device__ __forceinline__ uint32_t tonemap_pixel(const float4 p, bool gamma)
{
    if (p.w == 0.f) return 255u << 24;
    const float r = p.x / p.w, g = p.y / p.w, b = p.z / p.w;
    if (!gamma) return (255u << 24) | to_u32(r * 255) | (to_u32(g * 255) << 8) | (to_u32(b * 255) << 16);
    // quotients that are exact: for counts whose reciprocal is no normal number
    return (255u << 24) | srgb_byte(r, 1.0f, 1.0f) | (srgb_byte(g, 1.0f, 1.0f) << 8) | (srgb_byte(b, 1.0f, 1.0f) << 16);
}

// kPixels neighbouring columns per thread, each a coalesced load of its own, so
// that a thread has several pixels in flight; bound by memory (16 bytes in, 4 out
// per pixel) and the launch. 1 / 2 / 4 pixels: 1080p 12.3 / 10.3 / 11.3 us, 3840x2160
// 40.8 / 32.8 / 34.9 us (0.75 of the measured HBM rate). With three divisions per
// pixel, one pixel per thread: 16.5 and 58.3 us.
constexpr int kPixels = 2;
template <bool GAMMA>
__global__ void __launch_bounds__(128) k_tonemap(const float4 *__restrict__ accum, int32_t w, int32_t h, uint32_t *__restrict__ out)
{
    const int x0 = blockIdx.x * (128 * kPixels) + threadIdx.x, y = blockIdx.y;
    float4 p[kPixels];
#pragma unroll
    for (int k = 0; k < kPixels; ++k) {
        const int x = x0 + 128 * k;
        if (x < w) p[k] = __ldcs(accum + x + (size_t)y * w);
    }
#pragma unroll
    for (int k = 0; k < kPixels; ++k) {
        const int x = x0 + 128 * k;
        if (x >= w) break;
        uint32_t v;
        if (GAMMA && p[k].w >= 1e-30f && p[k].w <= 1e30f) {
            float inv;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(p[k].w));
            v = (255u << 24) | srgb_byte(p[k].x, p[k].w, inv) | (srgb_byte(p[k].y, p[k].w, inv) << 8) |
                (srgb_byte(p[k].z, p[k].w, inv) << 16);
        } else {
            v = tonemap_pixel(p[k], GAMMA);
        }
        __stcs(out + x + (size_t)(h - y - 1) * w, v);
    }
}

__global__ void k_resolve(const float4 *__restrict__ accum, uint64_t n, float *__restrict__ rgb)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = accum[i];
    const bool any = p.w != 0.f;
    rgb[3 * i] = any ? p.x / p.w : 0.0f;
    rgb[3 * i + 1] = any ? p.y / p.w : 0.0f;
    rgb[3 * i + 2] = any ? p.z / p.w : 0.0f;
}

}  // namespace
}  // namespace dr

using namespace dr;

extern "C" {

dr_status dr_framebuffer_create(dr_context *ctx, int32_t width, int32_t height, dr_framebuffer **out)
{
    DR_CHECK_ARG(ctx && out && width > 0 && height > 0, "dr_framebuffer_create: bad argument");
    DR_CHECK_ARG(height <= 65535 && (uint64_t)width * (uint64_t)height < (1ull << 31),
                 "dr_framebuffer_create: image too large");
    *out = nullptr;
    DR_CUDA(cudaSetDevice(ctx->device));
    auto *fb = new (std::nothrow) dr_framebuffer;
    if (!fb) return fail(DR_ERR_OUT_OF_MEMORY, "host allocation failed");
    fb->ctx = ctx;
    fb->width = width;
    fb->height = height;
    const size_t n = (size_t)width * height;
    cudaError_t e;
    if ((e = dev_malloc(&fb->accum, n * sizeof(float4))) != cudaSuccess ||
        (e = dev_malloc(&fb->casts, n * sizeof(uint32_t))) != cudaSuccess ||
        (e = dev_malloc(&fb->pixels, n * sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMemset(fb->accum, 0, n * sizeof(float4))) != cudaSuccess ||
        (e = cudaMemset(fb->casts, 0, n * sizeof(uint32_t))) != cudaSuccess) {
        dr_framebuffer_destroy(fb);
        return cuda_fail(e, "dr_framebuffer_create");
    }
    *out = fb;
    return DR_OK;
}

dr_status dr_framebuffer_destroy(dr_framebuffer *fb)
{
    if (!fb) return DR_OK;
    cudaSetDevice(fb->ctx->device);
    cudaFree(fb->accum);
    cudaFree(fb->casts);
    cudaFree(fb->pixels);
    delete fb;
    return DR_OK;
}

dr_status dr_framebuffer_clear(dr_framebuffer *fb, void *stream)
{
    DR_CHECK_ARG(fb != nullptr, "dr_framebuffer_clear: NULL");
    DR_CUDA(cudaSetDevice(fb->ctx->device));
    const size_t n = (size_t)fb->width * fb->height;
    auto st = static_cast<cudaStream_t>(stream);
    DR_CUDA(cudaMemsetAsync(fb->accum, 0, n * sizeof(float4), st));
    DR_CUDA(cudaMemsetAsync(fb->casts, 0, n * sizeof(uint32_t), st));
    return DR_OK;
}

dr_status dr_framebuffer_device_buffers(dr_framebuffer *fb, float **accum_dev, uint32_t **casts_dev)
{
    DR_CHECK_ARG(fb != nullptr, "dr_framebuffer_device_buffers: NULL");
    if (accum_dev) *accum_dev = reinterpret_cast<float *>(fb->accum);
    if (casts_dev) *casts_dev = fb->casts;
    return DR_OK;
}

dr_status dr_framebuffer_read(dr_framebuffer *fb, float *accum_host, uint32_t *casts_host, uint64_t *total_casts)
{
    DR_CHECK_ARG(fb != nullptr, "dr_framebuffer_read: NULL");
    DR_CUDA(cudaSetDevice(fb->ctx->device));
    const size_t n = (size_t)fb->width * fb->height;
    DR_CUDA(cudaDeviceSynchronize());
    if (accum_host) DR_CUDA(cudaMemcpy(accum_host, fb->accum, n * sizeof(float4), cudaMemcpyDeviceToHost));
    if (casts_host || total_casts) {
        std::vector<uint32_t> tmp;
        uint32_t *dst = casts_host;
        if (!dst) {
            tmp.resize(n);
            dst = tmp.data();
        }
        DR_CUDA(cudaMemcpy(dst, fb->casts, n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        if (total_casts) {
            uint64_t t = 0;
            for (size_t i = 0; i < n; ++i) t += dst[i];
            *total_casts = t;
        }
    }
    return DR_OK;
}

dr_status dr_tonemap(const float *accum_dev, int32_t width, int32_t height, int32_t gamma_corrected,
                     uint32_t *rgba_dev, void *stream)
{
    DR_CHECK_ARG(accum_dev && rgba_dev && width > 0 && height > 0, "dr_tonemap: bad argument");
    DR_CHECK_ARG(height <= 65535 && (uint64_t)width * (uint64_t)height < (1ull << 31), "dr_tonemap: image too large");
    DR_CHECK_ARG(((uintptr_t)accum_dev & 15) == 0, "dr_tonemap: accum_dev must be 16-byte aligned");
    // (unsigned: widths up to 2^31 - 1 are accepted)
    const dim3 grid(((unsigned)width + 128 * kPixels - 1) / (128 * kPixels), height);
    const auto st = static_cast<cudaStream_t>(stream);
    const auto *accum = reinterpret_cast<const float4 *>(accum_dev);
    if (gamma_corrected) k_tonemap<true><<<grid, 128, 0, st>>>(accum, width, height, rgba_dev);
    else k_tonemap<false><<<grid, 128, 0, st>>>(accum, width, height, rgba_dev);
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_resolve(const float *accum_dev, int32_t width, int32_t height, float *rgb_dev, void *stream)
{
    DR_CHECK_ARG(accum_dev && rgb_dev && width > 0 && height > 0, "dr_resolve: bad argument");
    DR_CHECK_ARG(((uintptr_t)accum_dev & 15) == 0, "dr_resolve: accum_dev must be 16-byte aligned");
    const uint64_t n = (uint64_t)width * (uint64_t)height;
    k_resolve<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4 *>(accum_dev), n, rgb_dev);
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_framebuffer_write_pfm(dr_framebuffer *fb, const char *path)
{
    DR_CHECK_ARG(fb && path, "dr_framebuffer_write_pfm: NULL");
    DR_CUDA(cudaSetDevice(fb->ctx->device));
    const size_t n = (size_t)fb->width * fb->height;
    float *rgb = nullptr;
    DR_CUDA(dev_malloc(&rgb, n * 3 * sizeof(float)));
    std::vector<float> host(n * 3);
    dr_status st = dr_resolve(reinterpret_cast<const float *>(fb->accum), fb->width, fb->height, rgb, nullptr);
    cudaError_t e = st == DR_OK ? cudaMemcpy(host.data(), rgb, n * 3 * sizeof(float), cudaMemcpyDeviceToHost)
                                : cudaSuccess;
    cudaFree(rgb);
    if (st != DR_OK) return st;
    if (e != cudaSuccess) return cuda_fail(e, "dr_framebuffer_write_pfm");
    FILE *f = fopen(path, "wb");
    if (!f) return fail(DR_ERR_INVALID_ARGUMENT, "dr_framebuffer_write_pfm: cannot open %s", path);
    // PFM header: colour, width height, negative scale = little-endian samples
    const int hdr = fprintf(f, "PF\n%d %d\n-1.0\n", fb->width, fb->height);
    uint32_t probe = 1;
    const bool little = *reinterpret_cast<unsigned char *>(&probe) == 1;
    bool ok = hdr > 0;
    if (ok && little) {
        ok = fwrite(host.data(), sizeof(float), host.size(), f) == host.size();
    } else if (ok) {
        for (size_t i = 0; ok && i < host.size(); ++i) {
            uint32_t b;
            memcpy(&b, &host[i], 4);
            const unsigned char le[4] = {(unsigned char)b, (unsigned char)(b >> 8), (unsigned char)(b >> 16),
                                         (unsigned char)(b >> 24)};
            ok = fwrite(le, 1, 4, f) == 4;
        }
    }
    ok = (fclose(f) == 0) && ok;
    if (!ok) return fail(DR_ERR_INVALID_ARGUMENT, "dr_framebuffer_write_pfm: writing %s failed", path);
    return DR_OK;
}

dr_status dr_framebuffer_tonemap(dr_framebuffer *fb, int32_t gamma_corrected, uint32_t *rgba_host)
{
    DR_CHECK_ARG(fb && rgba_host, "dr_framebuffer_tonemap: NULL");
    DR_CUDA(cudaSetDevice(fb->ctx->device));
    const dr_status st = dr_tonemap(reinterpret_cast<const float *>(fb->accum), fb->width, fb->height,
                                    gamma_corrected, fb->pixels, nullptr);
    if (st != DR_OK) return st;
    DR_CUDA(cudaMemcpy(rgba_host, fb->pixels, (size_t)fb->width * fb->height * sizeof(uint32_t),
                       cudaMemcpyDeviceToHost));
    return DR_OK;
}

dr_status dr_alias_build_host(dr_context *ctx, const float *w, uint32_t n, dr_alias_entry *out, int32_t mode)
{
    DR_CHECK_ARG(ctx != nullptr, "dr_alias_build_host: ctx is NULL");
    DR_CHECK_ARG(n == 0 || (w && out), "dr_alias_build_host: NULL buffer");
    if (n == 0) return DR_OK;
    DR_CUDA(cudaSetDevice(ctx->device));
    float *dw = nullptr;
    dr_alias_entry *dt = nullptr;
    DR_CUDA(dev_malloc(&dw, (size_t)n * sizeof(float)));
    cudaError_t e = dev_malloc(&dt, (size_t)n * sizeof(dr_alias_entry));
    if (e == cudaSuccess) e = cudaMemcpy(dw, w, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
    dr_status st = DR_OK;
    if (e == cudaSuccess) {
        st = dr_alias_build(ctx, dw, n, dt, mode, nullptr);
        if (st == DR_OK) e = cudaMemcpy(out, dt, (size_t)n * sizeof(dr_alias_entry), cudaMemcpyDeviceToHost);
    }
    cudaFree(dw);
    cudaFree(dt);
    if (e != cudaSuccess) return cuda_fail(e, "dr_alias_build_host");
    return st;
}

}  // extern "C"
