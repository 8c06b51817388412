// forces_ref.cu -- per-particle stack traversal with the reference's
// opening test (src/kernels/physics_kernels.py:14-153).
//
// One warp per group of consecutive targets, one shared stack (k_forces_walk).
// The opening test (x-extent, clamped to `box` above box/2, against theta^2 d^2
// with d the per-axis minimum image of the CoM) and the silent drop of both
// children when a target's 64-entry stack has fewer than two free slots are the
// reference's; the drop is also reported as CNB_FLAG_STACK_OVERFLOW.
//
// T = double follows the float64 arithmetic compiled Numba gives the
// reference (float32 node data, `round()` promoting the displacement);
// T = float is the float32 form.  The reference's shared-memory copy of the
// top 256 nodes only mirrors node data and is not needed for the result.
#include <type_traits>

#include "grouped.cuh"

namespace cnb {

// dx -= round(dx) of physics_kernels.py:118-120.  The float32 difference d minus
// its nearest integer is exact in float32 (a multiple of d's own ulp below 1/2),
// so the float64 form converts the result instead of rounding in float64.
template <typename T>
__device__ __forceinline__ T min_image(float d) {
    return (T)(d - rintf(d));
}

// q^(-3/2); in float32 q is at least kMinSoft2
__device__ __forceinline__ double inv_r3(double q) {
    const double r = rsqrt(q);
    return r * r * r;
}
__device__ __forceinline__ float inv_r3(float q) {
    const float r = rsqrt_normal(q);
    return r * r * r;
}

// The tree a walk reads: the reference's node arrays, or (rec not null) the
// 32-byte records of cnb_pack_nodes with the same values, one sector a node
// where the arrays take seven.
template <typename T>
struct RefTree {
    const int2 *children;
    const float *n_mass, *n_com, *n_min, *n_max;
    const float4 *rec;
    T theta_sq, G, soft2, box;
    int64_t m_nodes;
};

struct RefNode {
    float4 com;  // (com, mass)
    float sx;    // x-extent, before the clamp
    int2 ch;
};

template <bool TABLE, typename T>
__device__ __forceinline__ RefNode load_node(const RefTree<T> &R, int64_t v) {
    RefNode q;
    if (TABLE) {
        q.com = __ldg(R.rec + 2 * v);
        const float4 S = __ldg(R.rec + 2 * v + 1);
        q.sx = S.x;
        q.ch = make_int2(__float_as_int(S.z), __float_as_int(S.w));
    } else {
        q.com = make_float4(__ldg(R.n_com + 3 * v), __ldg(R.n_com + 3 * v + 1),
                            __ldg(R.n_com + 3 * v + 2), __ldg(R.n_mass + v));
        q.sx = __ldg(R.n_max + 3 * v) - __ldg(R.n_min + 3 * v);
        q.ch = __ldg(R.children + v);
    }
    return q;
}

// One body's depth-first walk with the reference's 64-entry stack: what a
// group falls back to when its shared walk could differ from it (a path of 63
// levels, where the reference may drop children, or a full shared stack).
template <bool TABLE, typename T>
__device__ __noinline__ void walk_one(const RefTree<T> &R, int32_t root, float x, float y, float z,
                                      T &ax, T &ay, T &az, bool &overflow, bool &bad) {
    ax = ay = az = 0;
    int32_t stack[64];
    int top = 0;
    stack[top++] = root;
    const T half_box = R.box * (T)0.5;
    int64_t visits = 0;
    while (top > 0) {
        // a valid tree visits every node at most once per target
        if (++visits > R.m_nodes) {
            bad = true;
            break;
        }
        const int32_t node = stack[--top];
        if (node < 0 || node >= R.m_nodes) {
            bad = true;
            continue;
        }
        const RefNode q = load_node<TABLE>(R, node);
        if (q.com.w <= 0.f) continue;
        const T dx = min_image<T>(q.com.x - x);
        const T dy = min_image<T>(q.com.y - y);
        const T dz = min_image<T>(q.com.z - z);
        const T d2 = dx * dx + dy * dy + dz * dz;
        bool use_node = (q.ch.x == -1);
        if (!use_node) {
            const T sx = ((T)q.sx > half_box) ? R.box : (T)q.sx;
            use_node = (sx * sx) < (R.theta_sq * d2);
        }
        if (use_node) {
            if (d2 > (T)1e-7) {
                const T f = R.G * (T)q.com.w * inv_r3(d2 + R.soft2);
                ax += f * dx;
                ay += f * dy;
                az += f * dz;
            }
        } else if (top + 1 < 64) {
            if (q.ch.x != -1) stack[top++] = q.ch.y;
            if (q.ch.y != -1) stack[top++] = q.ch.x;
        } else {
            overflow = true;
        }
    }
}

// A warp walks the tree once for GROUP consecutive targets.  A thread with a
// stack of its own reads ten words of a node of its own at every step and
// waits for them; neighbouring targets meet nearly the same nodes, so here a
// stack entry is a node and the set of the group's targets that reached it.
// Up to 32 entries are popped at a time and each lane fetches one node, all
// fetches in flight together; then the entries are applied, 32 / GROUP at a
// time, lane l holding target l % GROUP and taking entry l / GROUP of the
// step.  A target is tested against exactly the nodes its own walk would
// visit, with its own arithmetic; only the order of its sums differs.
//
// The reference's stack can be full only below 63 open levels (after a pop at
// depth d a walk holds at most d entries), so a group that opens a node at
// depth 63, or whose shared stack is full, starts over with walk_one, drops
// included; cyclic trees end there too.
//
// EXACT (T = float): the reference's float64 decisions on float32 forces, as
// forces_exact.cu makes them (the test in float64 inside the band [lo, hi]
// around s^2 / theta^2), without the reference's stack limit: the form the
// grouped traversal takes on small systems (CNB_EXACT_WALK_BODIES).
//
// Bound by the instructions of a step (about 40 for 32 pairs in float32); small
// counts by the latency of the fetches, one round of 32 after the other.  One
// thread per target against this, same values: float32 2 097 152 targets theta
// 0.5 41.7 -> 6.8 ms, 32 768 with the reference's scattered keys 48.0 -> 3.9 ms;
// float64 2 097 152 37.3 -> 11.4 ms, 5 000 of 64 000 840 -> 80 us.
//
// The stack never fills on a radix tree.  A popped entry leaves at most one more
// than it took, so popping a part of what is free below kRefDeep keeps rounds of
// several entries below it; from there on a round pops one, and a depth-first
// walk holds at most an entry a level more.  The levels of a tree over 64-bit
// keys, runs of equal ones split by index, are at most 64 + 32: the kRefDeep
// entries kept for it are more.  Only a caller's own, deeper tree can fill the stack.
//
// A full stack is slow, though: rounds of one node.  Walks at small angles open
// far more, and on deep trees fill 512 entries, so EXACT takes 848 below theta
// 0.4 (seven blocks an SM; 1024 leave six), and a sixteenth of the free ones a
// round instead of a quarter (us, 512 / 848 entries / the faster bucket shape; a
// cusp of 64 levels, then an even state): 5 000 bodies theta 0.1 1313 / 262 / 279, 170 /
// 168 / 451, theta 0.3 70 / 70 / 136, 63 / 64 / 229; 20 000 theta 0.1 5162 / 1292 / 868, 1012 /
// 1120 / 1387, theta 0.2 2326 / 590 / 497, 485 / 547 / 750, theta 0.3 1048 / 229 / 313, 236 /
// 260 / 393.  30 000 bodies with 1024 entries against buckets: theta 0.2 702 / 551, 907 / 870,
// theta 0.3 334 / 315, 426 / 451: the line between lies at 24 576
// (CNB_EXACT_WALK_BODIES_SMALL_ANGLE).
constexpr int kRefWarps = 4;
constexpr int kRefDeep = 128;
constexpr int kRefDepth = 63;
static_assert(kRefDeep > 64 + 32, "a level each for a depth-first walk");

// What a step reads of an entry, two 128-bit words: (com, w) and
//   float:  (G m, sx^2 or -1 for a leaf, targets, 0)
//   EXACT:  (lo, hi, s, targets), w the mass
//   double: (sx^2 or -1, G m), w the targets
template <int STACK, bool DEPTH>
struct WalkSmem {
    int2 stack[STACK];  // (node, targets)
    float4 node[32];
    float4 more[32];
    uint8_t depth[DEPTH ? STACK : 1];
};

// The rare part of an EXACT test: d^2 inside the band around s^2 / theta^2 or
// around the cut, both then decided in float64 (bit 0: accepted, bit 1: beyond the cut).
static __device__ __noinline__ int decide_f64(float s, double theta_sq, float dx, float dy, float dz) {
    const double d2 = (double)dx * dx + (double)dy * dy + (double)dz * dz;
    return ((double)s * (double)s < theta_sq * d2 ? 1 : 0) | (d2 > 1e-7 ? 2 : 0);
}

// STACK: entries of a warp's shared stack
template <typename T, int GROUP, bool TABLE, bool EXACT, int STACK>
__global__ void __launch_bounds__(kRefWarps * 32) k_forces_walk(
    const float *__restrict__ px, const float *__restrict__ py, const float *__restrict__ pz,
    RefTree<T> R, double theta_sq, float *__restrict__ force, const int32_t *__restrict__ root_idx,
    int32_t root_node, int64_t off, int64_t count, unsigned long long *stats, int32_t *max_stack,
    int32_t *status) {
    constexpr int SLOTS = 32 / GROUP;
    constexpr uint32_t kGroupMask = GROUP == 32 ? 0xffffffffu : (1u << (GROUP % 32)) - 1u;
    __shared__ WalkSmem<STACK, !EXACT> smem[kRefWarps];
    const int lane = threadIdx.x & 31;
    WalkSmem<STACK, !EXACT> &S = smem[threadIdx.x >> 5];
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t first = (blockIdx.x * (int64_t)kRefWarps + (threadIdx.x >> 5)) * GROUP;
    if (first >= count) return;
    const int slot = lane / GROUP, b = lane % GROUP;
    const int members = (int)(count - first < GROUP ? count - first : GROUP);
    const int64_t i = off + first + (b < members ? b : 0);
    const float x = px[i], y = py[i], z = pz[i];
    const bool owner = slot == 0 && b < members;
    if (owner && !(isfinite(x) && isfinite(y) && isfinite(z))) set_flag(status, CNB_FLAG_NONFINITE);
    const T half_box = R.box * (T)0.5;
    const float inv_th2 = 1.f / (float)theta_sq;
    const int32_t root = root_idx ? __ldg(root_idx) : root_node;
    T ax = 0, ay = 0, az = 0;
    bool overflow = false, bad = false, alone = false, full = false;
    int top = 1, deepest = 1;
    int64_t popped = 0;
    uint32_t n_acc = 0;
    if (lane == 0) {
        S.stack[0] = make_int2(root, (int)(members == 32 ? 0xffffffffu : (1u << members) - 1u));
        if (!EXACT) S.depth[0] = 0;
    }
    __syncwarp();
    while (top > 0) {
        // fewer as the stack fills, down to a depth-first walk
        const int room = (STACK - kRefDeep - top) >> (STACK > 512 ? 4 : 2);
        const int k = min(top, min(32, room > 1 ? room : 1));
        top -= k;
        popped += k;
        int2 ch = make_int2(-1, -1);
        uint32_t mask = 0;
        int depth = 0;
        if (lane < k) {
            const int2 e = S.stack[top + lane];
            if (!EXACT) depth = S.depth[top + lane];
            float4 N = make_float4(0.f, 0.f, 0.f, 0.f);
            T size2 = (T)-1;
            float2 band = make_float2(-1.f, -1.f);
            if (e.x < 0 || e.x >= R.m_nodes) {
                bad = true;
            } else {
                const RefNode q = load_node<TABLE>(R, e.x);
                N = q.com;
                ch = q.ch;
                if (!(N.w <= 0.f)) mask = (uint32_t)e.y;  // physics_kernels.py:114
                const T sx = ((T)q.sx > half_box) ? R.box : (T)q.sx;
                if (EXACT) {
                    const float s2 = (float)(sx * sx) * inv_th2;
                    size2 = sx;
                    if (ch.x != -1) band = make_float2(s2 * (1.f - kRelMargin), s2 * (1.f + kRelMargin));
                } else if (ch.x != -1) {
                    size2 = sx * sx;
                }
            }
            const float bits = __uint_as_float(mask);
            if constexpr (sizeof(T) == 8) {
                S.node[lane] = make_float4(N.x, N.y, N.z, bits);
                reinterpret_cast<double2 *>(S.more)[lane] = make_double2(size2, R.G * (T)N.w);
            } else {
                S.node[lane] = N;
                S.more[lane] = EXACT ? make_float4(band.x, band.y, (float)size2, bits)
                                     : make_float4((float)R.G * N.w, (float)size2, bits, 0.f);
            }
        }
        __syncwarp();
        uint32_t opened = 0;
        for (int j0 = 0; j0 < k; j0 += SLOTS) {
            const int j = j0 + slot;
            bool open = false;
            if (SLOTS == 1 || j < k) {
                const float4 N = S.node[j];
                const T dx = min_image<T>(N.x - x);
                const T dy = min_image<T>(N.y - y);
                const T dz = min_image<T>(N.z - z);
                const T d2 = dx * dx + dy * dy + dz * dz;
                if constexpr (sizeof(T) == 8) {
                    const double2 M = reinterpret_cast<const double2 *>(S.more)[j];
                    const bool in = (__float_as_uint(N.w) >> b) & 1u;
                    const bool use = M.x < 0.0 || M.x < R.theta_sq * d2;
                    open = in && !use;
                    if (in && use && d2 > 1e-7) {
                        const T f = M.y * inv_r3(d2 + R.soft2);
                        ax += f * dx;
                        ay += f * dy;
                        az += f * dz;
                    }
                } else {
                    const float4 M = S.more[j];
                    const bool in = (__float_as_uint(EXACT ? M.w : M.z) >> b) & 1u;
                    bool use, far;
                    if (EXACT) {
                        use = d2 > M.y;
                        far = d2 > kCutHi;
                        if (in && ((!use && !(d2 < M.x)) || (!far && !(d2 < kCutLo)))) {
                            const int r = decide_f64(M.z, theta_sq, dx, dy, dz);
                            if (!use && !(d2 < M.x)) use = r & 1;
                            if (!far && !(d2 < kCutLo)) far = r & 2;
                        }
                        n_acc += in && use;
                    } else {
                        use = M.y < 0.f || M.y < R.theta_sq * d2;
                        far = d2 > 1e-7f;
                    }
                    open = in && !use;
                    // the factor of every lane, the sums only of those that use the node
                    const T f = (EXACT ? N.w : M.x) * inv_r3(d2 + R.soft2);
                    if (in && use && far) {
                        ax += f * dx;
                        ay += f * dy;
                        az += f * dz;
                    }
                }
            }
            const uint32_t o = __ballot_sync(0xffffffffu, open);
            const int mine = lane - j0;  // this lane's own entry, if the step held it
            if (mine >= 0 && mine < SLOTS) opened = (o >> (mine * GROUP)) & kGroupMask;
        }
        // children of the opened entries, in the reference's push order
        const bool p1 = opened && ch.x != -1, p2 = opened && ch.y != -1;
        const uint32_t m1 = __ballot_sync(0xffffffffu, p1), m2 = __ballot_sync(0xffffffffu, p2);
        const int pushed = __popc(m1) + __popc(m2);
        if (top + pushed > STACK || popped > R.m_nodes ||
            (!EXACT && __any_sync(0xffffffffu, opened && depth >= kRefDepth))) {
            alone = true;
            full = top + pushed > STACK;
            break;
        }
        int at = top + __popc(m1 & lt) + __popc(m2 & lt);
        if (p1) {
            S.stack[at] = make_int2(ch.y, (int)opened);
            if (!EXACT) S.depth[at] = (uint8_t)(depth + 1);
            ++at;
        }
        if (p2) {
            S.stack[at] = make_int2(ch.x, (int)opened);
            if (!EXACT) S.depth[at] = (uint8_t)(depth + 1);
        }
        top += pushed;
        deepest = max(deepest, top);
        __syncwarp();
    }
    if (alone && EXACT) {
        // more visits than nodes: no tree; a full stack: the node set is incomplete
        if (lane == 0) set_flag(status, full ? CNB_FLAG_LIST_OVERFLOW : CNB_FLAG_BAD_TOPOLOGY);
    }
    if (alone && !EXACT) {
        if (owner) walk_one<TABLE, T>(R, root, x, y, z, ax, ay, az, overflow, bad);
    } else {
#pragma unroll
        for (int o = GROUP; o < 32; o <<= 1) {
            ax += __shfl_xor_sync(0xffffffffu, ax, o);
            ay += __shfl_xor_sync(0xffffffffu, ay, o);
            az += __shfl_xor_sync(0xffffffffu, az, o);
        }
    }
    if (overflow) set_flag(status, CNB_FLAG_STACK_OVERFLOW);
    if (bad) set_flag(status, CNB_FLAG_BAD_TOPOLOGY);
    if (EXACT) {
        const uint32_t acc = __reduce_add_sync(0xffffffffu, n_acc);
        if (lane == 0) {
            if (stats) {
                atomicAdd(stats, (unsigned long long)acc);
                atomicAdd(stats + 1, (unsigned long long)popped);
                atomicAdd(stats + 2, (unsigned long long)acc);
            }
            atomicMax(max_stack, deepest);
        }
    }
    if (!owner) return;
    const T scale = EXACT ? R.G : (T)1;
    const float fx = (float)(scale * ax), fy = (float)(scale * ay), fz = (float)(scale * az);
    force[3 * i] = fx;
    force[3 * i + 1] = fy;
    force[3 * i + 2] = fz;
    if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) set_flag(status, CNB_FLAG_NONFINITE);
}

template <typename T, int GROUP, bool TABLE, bool EXACT, int STACK>
static int launch_walk(const float *px, const float *py, const float *pz, const RefTree<T> &R,
                       double theta_sq, float *force, const int32_t *root_idx, int32_t root_node,
                       int64_t off, int64_t count, unsigned long long *stats, int32_t *max_stack,
                       int32_t *status, cudaStream_t st) {
    const int64_t per_block = (int64_t)kRefWarps * GROUP;
    const int64_t grid = (count + per_block - 1) / per_block;
    if (grid > INT32_MAX) return CNB_E_TOO_LARGE;
    k_forces_walk<T, GROUP, TABLE, EXACT, STACK><<<(unsigned)grid, kRefWarps * 32, 0, st>>>(
        px, py, pz, R, theta_sq, force, root_idx, root_node, off, count, stats, max_stack, status);
    return launch_status();
}

template <typename T, bool TABLE, bool EXACT, int STACK = 512>
static int forces_walk(const float *px, const float *py, const float *pz, const RefTree<T> &R,
                       double theta_sq, float *force, const int32_t *root_idx, int32_t root_node,
                       int64_t off, int64_t count, unsigned long long *stats, int32_t *max_stack,
                       int32_t *status, cudaStream_t st) {
    const auto go = [&](auto group) {
        return launch_walk<T, decltype(group)::value, TABLE, EXACT, STACK>(
            px, py, pz, R, theta_sq, force, root_idx, root_node, off, count, stats, max_stack, status, st);
    };
    // A smaller group shares less (more node fetches and tests in all) but gives more warps, and
    // below a few thousand warps a pass lasts as long as one warp's chain of fetches.  Measured
    // (us, groups of 2 / 4 / 8): float32 8 192 targets 51 / 55 / 71, 12 000 76 / 67 / 81, 24 576
    // 129 / 112 / 109, 131 072 635 / 464 / 424; float64 (a test costs more there, so wasted lanes
    // weigh more) 12 000 90 / 92 / 120, 48 000 291 / 261 / 293, 65 536 405 / 356 / 369, 131 072
    // 801 / 675 / 671; EXACT 10 000 55 / 57 / 81, 12 000 69 / 62 / 87, 32 768 146 / 126 / 129, 65 536
    // 304 / 251 / 256, 98 000 409 / 331 / 329.  Groups of 8 / 32: float32 300 007 1033 / 1015,
    // 2 097 152 7632 / 6775; float64 300 007 1563 / 1823, 2 097 152 11504 / 11350.
    if (count <= 10240) return go(std::integral_constant<int, 2>());
    if (EXACT || count <= (sizeof(T) == 8 ? 65536 : 24576)) return go(std::integral_constant<int, 4>());
    if constexpr (!EXACT) {
        if (count <= (sizeof(T) == 8 ? 1 << 20 : 1 << 18)) return go(std::integral_constant<int, 8>());
        return go(std::integral_constant<int, 32>());
    }
    return CNB_E_INVALID_ARG;
}

int launch_exact_walk(const GroupedParams &P, cudaStream_t st) {
    RefTree<float> R{};
    R.rec = P.rec;
    R.theta_sq = P.theta * P.theta;
    R.G = P.G;
    R.soft2 = normal_soft2(P.soft2);
    R.box = P.box;
    R.m_nodes = P.m_nodes;
    const auto walk = P.theta < 0.4f ? forces_walk<float, true, true, 848> : forces_walk<float, true, true>;
    return walk(P.px, P.py, P.pz, R, P.theta_sq, P.force, nullptr, P.root, 0, P.n, P.stats, P.ws + 2, P.status,
                st);
}

template <typename T, bool TABLE>
static int forces_ref(const float *px, const float *py, const float *pz, RefTree<T> R, float *force,
                      double theta, double G, double soft, double box, const int32_t *root_idx,
                      int64_t off, int64_t count, int64_t n, int32_t *status, cudaStream_t st) {
    R.theta_sq = (T)(theta * theta);
    R.G = (T)G;
    R.soft2 = (T)(soft * soft);
    if (sizeof(T) == 4) R.soft2 = normal_soft2((float)R.soft2);
    R.box = (T)box;
    R.m_nodes = 2 * n - 1;
    if (count > n - off) count = n - off;
    return forces_walk<T, TABLE, false>(px, py, pz, R, theta * theta, force, root_idx, 0, off, count,
                                        nullptr, nullptr, status, st);
}

}  // namespace cnb

using namespace cnb;

extern "C" int cnb_compute_forces(const float *px, const float *py, const float *pz,
                                  const int32_t *children, const float *n_mass,
                                  const float *n_com, const float *n_min, const float *n_max,
                                  float *force, double theta, double G, double soft, double box,
                                  const int32_t *root_idx, int64_t off, int64_t count, int64_t n,
                                  int precision, int32_t *status, void *stream) {
    if (n < 0 || off < 0 || count < 0) return CNB_E_INVALID_ARG;
    if (count == 0 || off >= n) return CNB_OK;
    if (!px || !py || !pz || !children || !n_mass || !n_com || !n_min || !n_max || !force ||
        !root_idx)
        return CNB_E_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(children) & 7) != 0) return CNB_E_INVALID_ARG;
    if (2 * n - 1 > (int64_t)INT32_MAX) return CNB_E_TOO_LARGE;
    const int2 *ch = reinterpret_cast<const int2 *>(children);
    cudaStream_t st = as_stream(stream);
    if (precision == CNB_PREC_F64)
        return forces_ref<double, false>(px, py, pz, {ch, n_mass, n_com, n_min, n_max}, force, theta,
                                         G, soft, box, root_idx, off, count, n, status, st);
    if (precision == CNB_PREC_F32)
        return forces_ref<float, false>(px, py, pz, {ch, n_mass, n_com, n_min, n_max}, force, theta,
                                        G, soft, box, root_idx, off, count, n, status, st);
    return CNB_E_INVALID_ARG;
}

extern "C" int cnb_compute_forces_table(const float *px, const float *py, const float *pz,
                                        const float *node_table, float *force, double theta,
                                        double G, double soft, double box, const int32_t *root_idx,
                                        int64_t off, int64_t count, int64_t n, int precision,
                                        int32_t *status, void *stream) {
    if (n < 0 || off < 0 || count < 0) return CNB_E_INVALID_ARG;
    if (count == 0 || off >= n) return CNB_OK;
    if (!px || !py || !pz || !node_table || !force || !root_idx) return CNB_E_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(node_table) & 15) != 0) return CNB_E_INVALID_ARG;
    if (2 * n - 1 > (int64_t)INT32_MAX) return CNB_E_TOO_LARGE;
    const float4 *rec = reinterpret_cast<const float4 *>(node_table);
    cudaStream_t st = as_stream(stream);
    if (precision == CNB_PREC_F64)
        return forces_ref<double, true>(px, py, pz, {nullptr, nullptr, nullptr, nullptr, nullptr, rec},
                                        force, theta, G, soft, box, root_idx, off, count, n, status, st);
    if (precision == CNB_PREC_F32)
        return forces_ref<float, true>(px, py, pz, {nullptr, nullptr, nullptr, nullptr, nullptr, rec},
                                       force, theta, G, soft, box, root_idx, off, count, n, status, st);
    return CNB_E_INVALID_ARG;
}
