// integrate_render.cu -- Hubble-drag kick/drift (physics_kernels.py:155-203)
// and the MVP density splat (render_kernels.py:12-47).
#include "common.cuh"

namespace cnb {

// physics_kernels.py:155-203: float64 kick and drift of float32 state, wrap
// by x - floor(x).  Explicit round-to-nearest operations (no contraction) so
// the result is the same on every compiler.
__global__ void __launch_bounds__(256) k_integrate(float *__restrict__ px, float *__restrict__ py,
                                                   float *__restrict__ pz, float *__restrict__ vx,
                                                   float *__restrict__ vy, float *__restrict__ vz,
                                                   const float *__restrict__ force, int64_t n,
                                                   double drag, double f_scale, double dt,
                                                   double drift) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        float *pp[3] = {px, py, pz};
        float *vv[3] = {vx, vy, vz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double v = __dadd_rn(__dmul_rn((double)vv[k][i], drag),
                                 __dmul_rn(__dmul_rn((double)__ldg(force + 3 * i + k), f_scale), dt));
            vv[k][i] = __double2float_rn(v);
            double p = __dadd_rn((double)pp[k][i], __dmul_rn(__dmul_rn(v, dt), drift));
            p = __dsub_rn(p, floor(p));
            pp[k][i] = __double2float_rn(p);
        }
    }
}

// ---------------------------------------------------------------- splat

// render_kernels.py:24-42: clip coordinates as float32 sums of float32
// products, w test / 1.0 / w / screen mapping in float64.  Returns the flat
// pixel index and the float32 weight 2.5 / w, or -1.
__device__ __forceinline__ int64_t splat_pixel(const float *m, float x, float y, float z,
                                               int width, int height, float *val) {
    float xc = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], x), __fmul_rn(m[1], y)),
                                   __fmul_rn(m[2], z)), m[3]);
    float yc = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[4], x), __fmul_rn(m[5], y)),
                                   __fmul_rn(m[6], z)), m[7]);
    float wc = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[12], x), __fmul_rn(m[13], y)),
                                   __fmul_rn(m[14], z)), m[15]);
    if (!((double)wc > 0.01)) return -1;
    double inv = __ddiv_rn(1.0, (double)wc);
    double sx = __dmul_rn(__dmul_rn(__dadd_rn(__dmul_rn((double)xc, inv), 1.0), 0.5), (double)width);
    double sy = __dmul_rn(__dmul_rn(__dsub_rn(1.0, __dmul_rn((double)yc, inv)), 0.5), (double)height);
    if (!(0.0 <= sx && sx < (double)width && 0.0 <= sy && sy < (double)height)) return -1;
    *val = __double2float_rn(__dmul_rn(2.5, inv));
    return (int64_t)sy * width + (int64_t)sx;
}

constexpr int kSplatThreads = 256;
constexpr int kSplatItems = 8;     // particles per thread
constexpr int kSplatBatch = 4;     // of them loaded together
constexpr int kSplatShare = 8;     // lanes on one pixel from which a warp adds them up first
constexpr int kSplatSlotBits = 12; // twice as many slots as a block has particles
constexpr int kSplatSlots = 1 << kSplatSlotBits;
constexpr uint32_t kSplatEmpty = 0xffffffffu;
static_assert(kSplatSlots >= 2 * kSplatThreads * kSplatItems, "a free slot is always found");

// A block's consecutive particles are added up in a shared-memory table of its
// pixels (open addressing), and each pixel goes to the grid with one atomic.
// Particles on one pixel have nearly the same weight, so adding them to the
// grid one after the other rounds in one direction, pixel after bright pixel:
// the block's sums keep the brightest pixel, which scales the whole frame, as
// exact as a block-wide tile of the grid does, and unlike that they need no
// bounding box, no passes over its dark pixels, and work for blocks whose
// pixels are far apart.
// Bound by the latency of the shared-memory atomics (half of the shared wavefronts;
// short scoreboard 4.8 stall cycles an issue, the most of any reason; issue 53 %,
// DRAM 11 %).  With the clear (us, a tile of the grid per
// block / one global atomic a particle / this): 2M particles on 1920x1080 41 /
// 18 / 31, 4M on 640x360 56 / 34 / 44, 300 007 on 1024x1024 23 / 8 / 16, 2M on
// 32x32 106 / 101 / 41, on 4x4 192 / 123 / 31.  The atomics a particle lose
// precision (frames of 32x32 pixels 8.3e-7 against 4.7e-7 from 64 bits, of 4x4
// 3.5e-6 against 7.6e-7); a slot as one 64-bit word takes 40 us on 1920x1080.
// A warp that piles up on a few pixels (a far camera, a small grid) is added up
// with shuffles before, while the first lane's pixel is shared by kSplatShare
// lanes or more.
__global__ void __launch_bounds__(kSplatThreads) k_splat(const float *__restrict__ px,
                                                         const float *__restrict__ py,
                                                         const float *__restrict__ pz,
                                                         float *__restrict__ grid, const float *__restrict__ mvp,
                                                         int64_t n, int width, int height, bool direct) {
    __shared__ __align__(16) uint32_t s_pix[kSplatSlots];
    __shared__ __align__(16) float s_sum[kSplatSlots];
    __shared__ float m[16];
    if (threadIdx.x < 16) m[threadIdx.x] = mvp[threadIdx.x];
    for (int k = threadIdx.x; k < kSplatSlots / 4; k += kSplatThreads) {
        reinterpret_cast<uint4 *>(s_pix)[k] = make_uint4(kSplatEmpty, kSplatEmpty, kSplatEmpty, kSplatEmpty);
        reinterpret_cast<float4 *>(s_sum)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const auto add = [&](int64_t pixel, float v) {
        if (direct) {
            atomicAdd(grid + pixel, v);
            return;
        }
        const uint32_t pix = (uint32_t)pixel;
        uint32_t at = (pix * 2654435761u) >> (32 - kSplatSlotBits);
        for (int tries = 0; tries < kSplatSlots; ++tries) {
            const uint32_t old = atomicCAS(s_pix + at, kSplatEmpty, pix);
            if (old == kSplatEmpty || old == pix) break;
            at = (at + 1) & (kSplatSlots - 1);
        }
        atomicAdd(s_sum + at, v);
    };
    const int lane = threadIdx.x & 31;
    const int64_t base = (int64_t)blockIdx.x * kSplatThreads * kSplatItems + threadIdx.x;
#pragma unroll
    for (int r0 = 0; r0 < kSplatItems; r0 += kSplatBatch) {
        float x[kSplatBatch], y[kSplatBatch], z[kSplatBatch];
#pragma unroll
        for (int r = 0; r < kSplatBatch; ++r) {
            const int64_t i = base + (int64_t)(r0 + r) * kSplatThreads;
            x[r] = i < n ? __ldcs(px + i) : 0.f;
            y[r] = i < n ? __ldcs(py + i) : 0.f;
            z[r] = i < n ? __ldcs(pz + i) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < kSplatBatch; ++r) {
            float val = 0.f;
            int64_t pix = base + (int64_t)(r0 + r) * kSplatThreads < n
                              ? splat_pixel(m, x[r], y[r], z[r], width, height, &val) : -1;
            for (uint32_t todo = __ballot_sync(0xffffffffu, pix >= 0); todo != 0u;) {
                const int lead = __ffs(todo) - 1;
                const int64_t p = __shfl_sync(0xffffffffu, pix, lead);
                const uint32_t same = __ballot_sync(0xffffffffu, pix == p);
                if (__popc(same) < kSplatShare) break;
                float sum = pix == p ? val : 0.f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane == lead) add(p, sum);
                if (pix == p) pix = -1;
                todo &= ~same;
            }
            if (pix >= 0) add(pix, val);
            __syncwarp();
        }
    }
    if (direct) return;
    __syncthreads();
    for (int k = threadIdx.x; k < kSplatSlots; k += kSplatThreads)
        if (s_pix[k] != kSplatEmpty) atomicAdd(grid + s_pix[k], s_sum[k]);
}

}  // namespace cnb

using namespace cnb;

extern "C" int cnb_integrate(float *px, float *py, float *pz, float *vx, float *vy, float *vz,
                             const float *force, int64_t n, double a, double H, double dt,
                             void *stream) {
    if (n < 0) return CNB_E_INVALID_ARG;
    if (n == 0) return CNB_OK;
    if (!px || !py || !pz || !vx || !vy || !vz || !force) return CNB_E_INVALID_ARG;
    const double drag = 1.0 - (H * dt);
    const double f_scale = 1.0 / a;
    const double drift = 1.0 / a;
    k_integrate<<<grid_for(n, 256, 148 * 16), 256, 0, as_stream(stream)>>>(
        px, py, pz, vx, vy, vz, force, n, drag, f_scale, dt, drift);
    return launch_status();
}

extern "C" int cnb_render_density(const float *px, const float *py, const float *pz,
                                  float *grid, const float *mvp, int64_t n, int width,
                                  int height, void *stream) {
    if (n < 0 || width <= 0 || height <= 0) return CNB_E_INVALID_ARG;
    if (n == 0) return CNB_OK;
    if (!px || !py || !pz || !grid || !mvp) return CNB_E_INVALID_ARG;
    const int64_t per_block = (int64_t)kSplatThreads * kSplatItems;
    const int64_t blocks = (n + per_block - 1) / per_block;
    if (blocks > INT32_MAX) return CNB_E_TOO_LARGE;
    // the block's table holds 32-bit pixels
    const bool direct = (int64_t)width * height >= (int64_t)kSplatEmpty;
    k_splat<<<(unsigned)blocks, kSplatThreads, 0, as_stream(stream)>>>(px, py, pz, grid, mvp, n,
                                                                      width, height, direct);
    return launch_status();
}
