// colorize.cu -- density grid -> RGB frame (src/utils/visualizer.py:115-171)
// in two kernels instead of ~20 elementwise launches: the grid's maximum,
// then one pass doing normalisation, gamma 2.2, the four-band
// colour map, the x1.3 gain, the clip and (optionally) the 8-bit packing of
// src/core/engine.py:139.  float32 throughout, as the reference's CuPy code.
#include "common.cuh"

namespace cnb {

// The grid's maximum (at least 0, NaN ignored); log1p(120 g) rises with g, so its
// maximum is taken of one value, where it is needed.  HBM/L2-bound: 4 bytes a
// pixel, four pixels a load.
__global__ void __launch_bounds__(256) k_grid_max(const float *__restrict__ grid, int64_t n, int64_t quads,
                                                  unsigned int *__restrict__ max_bits) {
    float m = 0.f;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t q = t; q < quads; q += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(grid)[q];
        m = fmaxf(fmaxf(m, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    }
    for (int64_t i = 4 * quads + t; i < n; i += (int64_t)gridDim.x * blockDim.x) m = fmaxf(m, grid[i]);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    // non-negative floats order like their bit patterns
    if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(max_bits, __float_as_uint(m));
}

// One pixel: normalisation by denom, gamma 2.2, the four bands, gain, clip.
__device__ __forceinline__ void colour(float v, float denom, float &r, float &g, float &b) {
    r = g = b = 0.f;
    if (v == 0.f) return;  // log1p(0) = 0: the first band's black (most of a frame)
    const float T1 = 0.6f, T2 = 0.72f, T3 = 0.82f;
    const float img = log1pf(v * 120.0f) / denom;
    const float val = powf(img, 2.2f);
    if (val <= T1) {
        b = (val / T1) * 0.8f;
    } else if (val <= T2) {
        const float t = (val - T1) / (T2 - T1);
        b = (1.0f - t) * 0.8f;
        g = t * 0.9f;
    } else if (val <= T3) {
        const float t = (val - T2) / (T3 - T2);
        g = 0.9f + t * 0.1f;
        r = t;
    } else {
        const float t = (val - T3) / (1.0f - T3);
        r = 1.0f;
        g = 1.0f - t;
    }
    r = fminf(fmaxf(r * 1.3f, 0.f), 1.f);
    g = fminf(fmaxf(g * 1.3f, 0.f), 1.f);
    b = fminf(fmaxf(b * 1.3f, 0.f), 1.f);
}

// (frame * 255).astype(uint8): truncation
__device__ __forceinline__ unsigned int byte_of(float c) { return (unsigned char)(c * 255.0f); }

// HBM-bound: 4 bytes in and 12 (+3) out a pixel.  Four pixels a thread where the
// arrays are aligned for it (`quads` of them: 128-bit loads and stores), the
// rest one by one; dark pixels skip the logarithm and the power.  1920x1080
// with 2M particles 15 -> 9.5 us, the maximum before it 9 -> 5.
__global__ void __launch_bounds__(256) k_colorize(const float *__restrict__ grid, int64_t n, int64_t quads,
                                                  const unsigned int *__restrict__ max_bits,
                                                  float *__restrict__ rgb,
                                                  unsigned char *__restrict__ rgb8) {
    const float denom = log1pf(__uint_as_float(*max_bits) * 120.0f) + 1e-9f;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t q = t; q < quads; q += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(grid)[q];
        float c[12];
        colour(v.x, denom, c[0], c[1], c[2]);
        colour(v.y, denom, c[3], c[4], c[5]);
        colour(v.z, denom, c[6], c[7], c[8]);
        colour(v.w, denom, c[9], c[10], c[11]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (rgb)
                reinterpret_cast<float4 *>(rgb)[3 * q + k] =
                    make_float4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
            if (rgb8)
                reinterpret_cast<unsigned int *>(rgb8)[3 * q + k] =
                    byte_of(c[4 * k]) | byte_of(c[4 * k + 1]) << 8 | byte_of(c[4 * k + 2]) << 16 |
                    byte_of(c[4 * k + 3]) << 24;
        }
    }
    for (int64_t i = 4 * quads + t; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float c[3];
        colour(grid[i], denom, c[0], c[1], c[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (rgb) rgb[3 * i + k] = c[k];
            if (rgb8) rgb8[3 * i + k] = (unsigned char)byte_of(c[k]);
        }
    }
}

}  // namespace cnb

extern "C" int cnb_colorize(const float *grid, int width, int height, float *rgb,
                            unsigned char *rgb8, unsigned int *scratch, void *stream) {
    if (width <= 0 || height <= 0 || !grid || !scratch || (!rgb && !rgb8)) return CNB_E_INVALID_ARG;
    const int64_t n = (int64_t)width * height;
    cudaStream_t st = cnb::as_stream(stream);
    CNB_CUDA(cudaMemsetAsync(scratch, 0, sizeof(unsigned int), st));
    auto at = [](const void *p, int align) { return (reinterpret_cast<uintptr_t>(p) & (align - 1)) == 0; };
    const int64_t g4 = at(grid, 16) ? n / 4 : 0;
    cnb::k_grid_max<<<cnb::grid_for(g4 ? g4 : n, 256, 148 * 8), 256, 0, st>>>(grid, n, g4, scratch);
    CNB_TRY(cnb::launch_status());
    const int64_t quads = at(rgb, 16) && at(rgb8, 4) ? g4 : 0;
    cnb::k_colorize<<<cnb::grid_for(quads ? quads : n, 256, 148 * 16), 256, 0, st>>>(grid, n, quads, scratch,
                                                                                   rgb, rgb8);
    return cnb::launch_status();
}
