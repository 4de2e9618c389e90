// resolve.cu -- MSAA resolve of a colour surface into a linear RGBA8 image.
//
// The reference's resolve (CudaSurface::resolveToScreen, CudaSurface.hpp:73)
// is commented out and would have drawn through GL. Here one thread per
// pixel averages the pixel's samples channel by channel, rounding half up:
// c = (sum of the S samples' channel + S/2) >> log2 S, and writes the pixel
// to a row-major image (one 32-bit word per pixel, R in the low byte as the
// surface words are). With one sample it only drops the 8x8 tile padding.
#include <cuda_runtime.h>

#include <cstdint>

#include "cudaraster.h"
#include "cudaraster/detail/launch.h"

namespace cr {
namespace {

// Channels R and B of a sample summed in the 16-bit lanes of `rb`, G and A in
// those of `ga`: a lane holds at most 8 * 255 + 4 < 2^16, so lanes never carry
// into each other, and the bits a right shift moves across a lane boundary are
// masked off.
struct SampleSum {
    uint32_t rb = 0, ga = 0;
    __device__ __forceinline__ void add(uint32_t c) {
        rb += c & 0x00FF00FFu;
        ga += (c >> 8) & 0x00FF00FFu;
    }
    template <int samplesLog2>
    __device__ __forceinline__ uint32_t average() const {
        constexpr uint32_t half = (uint32_t)((1 << samplesLog2) >> 1) * 0x00010001u;
        return (((rb + half) >> samplesLog2) & 0x00FF00FFu) | ((((ga + half) >> samplesLog2) & 0x00FF00FFu) << 8);
    }
};

// Surfaces at a 16-byte boundary (every torch or cudaMalloc allocation): four
// neighbouring pixels per thread, a 16-byte load per sample; a warp's 128
// pixels pass through shared memory, so that its stores are whole lines
// wherever the output's rows start. HBM-bound: a 4x 3839x2159 surface 28.7 us,
// 33.2 with the kernel below (a thread per pixel, 4-byte loads, which left too
// few bytes in flight).
template <int samplesLog2>
__global__ void __launch_bounds__(256) resolveWideKernel(const uint32_t* __restrict__ color, int width, int height,
                                                         int64_t rowWords, uint32_t* __restrict__ out,
                                                         int64_t outRowWords) {
    __shared__ uint4 s_out[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = blockIdx.x * 128, y = blockIdx.y * 8 + warp;
    if (y >= height) return;
    constexpr int ns = 1 << samplesLog2;
    const int x = x0 + lane * 4;   // the surface's rows are padded to multiples of 8 pixels
    if (x < width) {
        const int64_t base = (int64_t)y * rowWords + (int64_t)(x >> 3) * 8 * ns + (x & 7);
        uint4 c[ns];
#pragma unroll
        for (int i = 0; i < ns; i++) c[i] = __ldg(reinterpret_cast<const uint4*>(color + base + i * 8));
        SampleSum a[4];
#pragma unroll
        for (int i = 0; i < ns; i++) {
            a[0].add(c[i].x);
            a[1].add(c[i].y);
            a[2].add(c[i].z);
            a[3].add(c[i].w);
        }
        s_out[warp][lane] = make_uint4(a[0].average<samplesLog2>(), a[1].average<samplesLog2>(),
                                       a[2].average<samplesLog2>(), a[3].average<samplesLog2>());
    }
    __syncwarp();
    const uint32_t* line = reinterpret_cast<const uint32_t*>(s_out[warp]);
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (x0 + k * 32 + lane < width) out[(int64_t)y * outRowWords + x0 + k * 32 + lane] = line[k * 32 + lane];
}

// Other surfaces: one thread per pixel; the sample count is a template
// parameter so the sample loads are unrolled and issued together.
template <int samplesLog2>
__global__ void resolveKernel(const uint32_t* __restrict__ color, int width, int height, int64_t rowWords,
                              uint32_t* __restrict__ out, int64_t outRowWords) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    constexpr int ns = 1 << samplesLog2;
    const int64_t base = (int64_t)y * rowWords + (int64_t)(x >> 3) * 8 * ns + (x & 7);
    SampleSum sum;
#pragma unroll
    for (int i = 0; i < ns; i++) sum.add(__ldg(&color[base + i * 8]));
    out[(int64_t)y * outRowWords + x] = sum.average<samplesLog2>();
}

template <int samplesLog2>
cudaError_t launchResolve(const uint32_t* color, int width, int height, int64_t rowWords, uint32_t* out,
                          int64_t outRowWords, cudaStream_t s) {
    if (((uintptr_t)color & 15) == 0)
        return launchKernel(resolveWideKernel<samplesLog2>, dim3((width + 127) / 128, (height + 7) / 8), 256, 0, s, false,
                            color, width, height, rowWords, out, outRowWords);
    return launchKernel(resolveKernel<samplesLog2>, dim3((width + 31) / 32, (height + 7) / 8), dim3(32, 8), 0, s, false,
                        color, width, height, rowWords, out, outRowWords);
}

}  // namespace
}  // namespace cr

extern "C" cr_status cr_resolve_color(const void* color, int32_t width, int32_t height, int32_t num_samples, void* out,
                                      int64_t out_row_bytes, void* stream) {
    if (!color || !out || width <= 0 || height <= 0 || width > CR_MAX_VIEWPORT || height > CR_MAX_VIEWPORT ||
        num_samples < 1 || num_samples > 8 || (num_samples & (num_samples - 1)) || out_row_bytes < (int64_t)width * 4 ||
        (out_row_bytes & 3))
        return CR_ERR_INVALID_ARGUMENT;
    int log2 = 0;
    while ((1 << log2) < num_samples) log2++;
    const int64_t rowWords = (int64_t)((width + 7) & ~7) * num_samples;
    const uint32_t* c = (const uint32_t*)color;
    uint32_t* o = (uint32_t*)out;
    const cudaStream_t s = (cudaStream_t)stream;
    const int64_t ow = out_row_bytes / 4;
    cudaError_t e;
    switch (log2) {
    case 0: e = cr::launchResolve<0>(c, width, height, rowWords, o, ow, s); break;
    case 1: e = cr::launchResolve<1>(c, width, height, rowWords, o, ow, s); break;
    case 2: e = cr::launchResolve<2>(c, width, height, rowWords, o, ow, s); break;
    default: e = cr::launchResolve<3>(c, width, height, rowWords, o, ow, s); break;
    }
    return e == cudaSuccess ? CR_OK : CR_ERR_CUDA;
}
