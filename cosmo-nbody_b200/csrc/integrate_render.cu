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
constexpr int kSplatItems = 2;  // particles per thread
constexpr int kSplatShare = 8;  // lanes on one pixel from which a warp adds them up first

// One global atomic per visible particle: a block's 2048 consecutive particles
// touch nearly as many pixels (400 thousand lit pixels of 2M particles at
// 1920x1080), so adding them up in a shared-memory tile first spared few atomics
// and cost a bounding box, two passes over the tile and its occupancy: 2M
// particles 35 against 14 us, 4M on 640x360 (73 a lit pixel) 51 against 33 with
// the clear.  What it did spare is the pile-up of a warp on a few pixels (a far
// camera, a small grid): there the warp's values are added up with shuffles,
// pixel by pixel while the first lane's pixel is shared by kSplatShare lanes or
// more (2M particles on 32x32 pixels 104 against 94 us, on 4x4 187 against 119).
__global__ void __launch_bounds__(kSplatThreads) k_splat(const float *__restrict__ px,
                                                         const float *__restrict__ py,
                                                         const float *__restrict__ pz,
                                                         float *__restrict__ grid, const float *__restrict__ mvp,
                                                         int64_t n, int width, int height) {
    __shared__ float m[16];
    if (threadIdx.x < 16) m[threadIdx.x] = mvp[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t base = (int64_t)blockIdx.x * kSplatThreads * kSplatItems + threadIdx.x;
    float x[kSplatItems], y[kSplatItems], z[kSplatItems];
#pragma unroll
    for (int r = 0; r < kSplatItems; ++r) {
        const int64_t i = base + (int64_t)r * kSplatThreads;
        x[r] = i < n ? __ldcs(px + i) : 0.f;
        y[r] = i < n ? __ldcs(py + i) : 0.f;
        z[r] = i < n ? __ldcs(pz + i) : 0.f;
    }
#pragma unroll
    for (int r = 0; r < kSplatItems; ++r) {
        float val = 0.f;
        int64_t pix = base + (int64_t)r * kSplatThreads < n
                          ? splat_pixel(m, x[r], y[r], z[r], width, height, &val) : -1;
        for (uint32_t todo = __ballot_sync(0xffffffffu, pix >= 0); todo != 0u;) {
            const int lead = __ffs(todo) - 1;
            const int64_t p = __shfl_sync(0xffffffffu, pix, lead);
            const uint32_t same = __ballot_sync(0xffffffffu, pix == p);
            if (__popc(same) < kSplatShare) break;
            float sum = pix == p ? val : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == lead) atomicAdd(grid + p, sum);
            if (pix == p) pix = -1;
            todo &= ~same;
        }
        if (pix >= 0) atomicAdd(grid + pix, val);
    }
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
    k_splat<<<(unsigned)blocks, kSplatThreads, 0, as_stream(stream)>>>(px, py, pz, grid, mvp, n,
                                                                      width, height);
    return launch_status();
}
