// forces_exact.cu -- the warp-per-bucket traversal with the reference's own
// opening decisions (src/kernels/physics_kernels.py:14-153, opening test
// :131-136): every body receives exactly the nodes its per-body stack walk
// accepts, in float32 arithmetic.
//
// One warp takes a bucket (a maximal subtree of at most 32*BPL bodies, lane l
// holding bodies l and l + 32).  Stack entries carry the set of the bucket's
// bodies that reached the node (a 64-bit mask: bit l of word b is body
// l + 32b); entries reached by the whole bucket sit on the main stack as
// plain node indices, the others on a second stack with their mask.  Each
// lane classifies one node against the bucket's box with the reference's
// test, sx^2 < theta^2 d^2 (sx the node's x-extent, set to the box above
// half a box; d the minimum-image distance from the body to the node's CoM):
//   every body of the mask accepts it   (sx^2 < theta^2 dmin^2)  -> list entry
//   every body of the mask opens it     (sx^2 > theta^2 dmax^2)  -> push children
//   the box cannot tell                                          -> per-body item
// with dmin / dmax the smallest / largest distance any point of the box can
// have to the CoM, widened by kBoxSlack and compared with a relative margin
// so that float32 rounding never decides.  Per-body items are evaluated by
// all lanes (each body its own d^2 and test, the force of the bodies that
// accept applied at once); the bodies that open the node push its children
// with their mask.  Leaves are accepted by every body that reaches them.
//
// Per body the float32 test reproduces the reference's float64 decision:
// the CoM difference fl32(c - x) is the reference's own float32 value, its
// minimum image d - rint(d) is exact in float32, and where the float32
// d^2 leaves sx^2 and theta^2 d^2 within kRelMargin of each other (or d^2
// within a band around the cut 1e-7) the test is redone in float64 like the
// reference.  The forces differ from the reference's only by float32 against
// float64 arithmetic and summation order.
//
// Lists: entries with one image for every body of their mask and out of the
// cut's reach go to the masked list (packed float2 for two bodies per lane, no
// image, no cut, the mass selected per body by the entry's mask; whole-bucket
// entries too: a list of their own saves them five instructions and costs
// every round more); every other accepted entry keeps the node's raw CoM and
// is applied with the per-pair minimum image, the cut and its mask.
// Per-body items carry the band [lo, hi] around s^2 / theta^2 inside which
// the float32 d^2 cannot decide.  Most are simple (87 % at 128^3): one image
// for every body, out of the cut's reach, and a CoM that shifts to that image
// exactly, so a round applies them first, without image, cut or flags; the
// others follow with the per-pair form.  Each lane keeps the node it
// classified, the mask of the bodies that accept it comes back to it, and the
// children of a round's items are pushed together after them.  Measured
// against one loop over flagged items (128^3, theta 0.5, 64-body buckets,
// two-level): 4.98 -> 4.74 ms; 32-body buckets, one level: 7.25 -> 6.72 ms.
//
// The node stacks live in shared memory (see kXWords); a bucket that would
// outgrow them in the main pass is walked again by a second launch with a
// larger region, so deep walks keep their exact node sets.
//
// Limit: the reference's 64-entry stack drops children when full
// (physics_kernels.py:143-149).  That happens only for trees deeper than
// about 63 levels; the exact walk has no such drop.
#include "grouped.cuh"

namespace cnb {

// The two node stacks of a warp share one region of XW words: entries
// reached by the whole bucket (one word, the node) grow up from word 0,
// entries reached by part of it (three words: node, mask low, mask high)
// grow down from the end.  A round pops no more entries than the free words
// can take back, so it is full until 160 words are left and narrows from there.
// A walk that goes on in rounds of fewer than kXLeast entries would crawl, so
// after kXNarrow of them (or without room for one) the main pass gives the
// bucket up: it marks the bucket's record and writes no force for it.  A second
// pass walks those buckets again with a region of kXWordsRedo words, by the main
// pass's rule up to where that gave up and in full rounds from there.  Its last
// kXDeep words are left to rounds of one entry, a depth-first walk: it takes at
// most five words where part of the bucket first opens a node and three a level
// from there, and a radix tree over 64-bit keys has at most 64 + 32 levels, so
// only a caller's own, deeper tree can overflow the region
// (CNB_FLAG_LIST_OVERFLOW).
//
// The main pass's region, by what a walk needs and what its words cost in warps
// and cache: at theta = 0.5 on 128^3 and 256^3 Zel'dovich and evolved states (two
// levels included) the deepest use is 607 words; cusps of 64 levels use 400 to
// 800 at theta 0.5 and above, 1200 to 1500 at 0.3, 2000 at 0.1.  Measured (us,
// regions of 640 / 864 / 1280 / 1536 / 2048 words): 500k Zel'dovich bodies theta
// 0.3 3960 / - / 4000 / 4140 / 4300, 120k bodies in a cusp, 64-body buckets, theta
// 0.5 880 / 555, theta 0.3 2370 / - / 1270 / 1340 / 1350, theta 0.25 - / - / 3010 / 1690,
// theta 0.1 9290 / - / 9720 / - / 5360; 16 boxes 1405 / 1450; 2M bodies theta 0.5 the same
// within 0.5 %.  Without the second pass's share (32 neighbouring records a warp,
// so that a cusp's buckets fell to a few warps) and the limit on narrow rounds
// 640 words for every angle took 14.5 ms at theta 0.3 and 82 ms at 0.1.
constexpr int kXWords = 640;        // one body a lane; several boxes
constexpr int kXWordsTwo = 864;     // two bodies a lane
constexpr int kXWordsWide = 1280;   // theta below 0.4
constexpr int kXWordsWidest = 2048; // theta below 0.25
constexpr int kXWordsRedo = 4096;   // the buckets a main pass gave up on
constexpr int kXLeast = 8, kXNarrow = 16, kXDeep = 320;
static_assert(kXDeep >= 5 + 3 * (64 + 32), "three words a level for a depth-first walk");
template <int XW> __device__ __forceinline__ int part_word(int k) { return XW - 3 * (k + 1); }

// per-warp shared memory: the masked list (packed for two bodies per lane), the
// per-pair list (one float4 per entry), the per-body items of one round, the
// two lists' masks and the stack region
template <int BPL> __host__ __device__ constexpr int exact_f4_per_warp() {
    return kGList * entry_width<BPL>() + kGList + 3 * 32;
}
constexpr int kExactMasksPerWarp = 2 * kGList;  // uint2

template <int BPL>
constexpr size_t exact_smem(int warps, int xw) {
    return (size_t)warps * (exact_f4_per_warp<BPL>() * sizeof(float4) +
                            kExactMasksPerWarp * sizeof(uint2) + xw * sizeof(int32_t));
}

// per-body item flags
constexpr int kItemWrap = 1;  // the CoM's minimum image can differ between the bucket's bodies
constexpr int kItemNear = 2;  // the item is close enough to the bucket for the cut to apply

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }

// d - rint(d) through the 1.5 * 2^23 rounding constant (|d| < 2^22): the
// reference's d - round(d), exact in float32 for |d| < 1
__device__ __forceinline__ float minus_image(float d) {
    return d - __fsub_rn(__fadd_rn(d, 12582912.f), 12582912.f);
}
__device__ __forceinline__ float2 minus_image2(float2 d) {
    const float2 rc = dup2(12582912.f), nrc = dup2(-12582912.f);
    return __ffma2_rn(__fadd2_rn(__fadd2_rn(d, rc), nrc), dup2(-1.f), d);
}

// Entry j of a list as the two packed float4 (x, x, y, y), (z, z, m, m) of the
// two-bodies-per-lane loop: stored so (put_entry), or SINGLE: stored once as
// (x, y, z, m) and duplicated here (the rarely filled per-pair list).
template <bool SINGLE>
__device__ __forceinline__ void entry_pair(const float4 *list, int j, float4 &a, float4 &b) {
    if (SINGLE) {
        const float4 e = list[j];
        a = make_float4(e.x, e.x, e.y, e.y);
        b = make_float4(e.z, e.z, e.w, e.w);
    } else {
        a = list[2 * j];
        b = list[2 * j + 1];
    }
}

// Masked list: cnt entries applied to the lane's bodies in the entry's mask.
// WRAP_CUT: raw CoM, one float4 per entry, with the per-pair minimum image
// and the cut; otherwise the CoM at the one image every body of the bucket
// sees, out of the cut's reach (two float4 per entry for two bodies per
// lane, as put_entry writes them).
template <int BPL, bool WRAP_CUT>
__device__ __forceinline__ void apply_masked(const float4 *list, const uint2 *masks, int cnt,
                                             int lane, const float (&x)[BPL], const float (&y)[BPL],
                                             const float (&z)[BPL], float soft2, float (&ax)[BPL],
                                             float (&ay)[BPL], float (&az)[BPL]) {
    const float cut = soft2 + 1e-7f;
    const uint32_t lane_bit = 1u << lane;
    if constexpr (BPL == 2) {
        const float2 nx = make_float2(-x[0], -x[1]), ny = make_float2(-y[0], -y[1]),
                     nz = make_float2(-z[0], -z[1]);
        const float2 s2 = dup2(soft2);
        float2 fx = make_float2(ax[0], ax[1]), fy = make_float2(ay[0], ay[1]),
               fz = make_float2(az[0], az[1]);
        // four entries at a time: loads, distances and masses first, then the
        // inverse cubes and the accumulation in list order
        int j = 0;
        for (; j + 4 <= cnt; j += 4) {
            float2 dx[4], dy[4], dz[4], w[4], q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float4 a, b;
                entry_pair<WRAP_CUT>(list, j + u, a, b);
                const uint2 mk = masks[j + u];
                dx[u] = __fadd2_rn(make_float2(a.x, a.y), nx);
                dy[u] = __fadd2_rn(make_float2(a.z, a.w), ny);
                dz[u] = __fadd2_rn(make_float2(b.x, b.y), nz);
                if (WRAP_CUT) {
                    dx[u] = minus_image2(dx[u]);
                    dy[u] = minus_image2(dy[u]);
                    dz[u] = minus_image2(dz[u]);
                }
                q[u] = __ffma2_rn(dx[u], dx[u], __ffma2_rn(dy[u], dy[u], __ffma2_rn(dz[u], dz[u], s2)));
                const bool u0 = (mk.x & lane_bit) != 0u, u1 = (mk.y & lane_bit) != 0u;
                w[u] = make_float2(u0 && (!WRAP_CUT || q[u].x > cut) ? b.z : 0.f,
                                   u1 && (!WRAP_CUT || q[u].y > cut) ? b.w : 0.f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 r = make_float2(rsqrt_normal(q[u].x), rsqrt_normal(q[u].y));
                const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(w[u], r), r), r);
                fx = __ffma2_rn(f, dx[u], fx);
                fy = __ffma2_rn(f, dy[u], fy);
                fz = __ffma2_rn(f, dz[u], fz);
            }
        }
        for (; j < cnt; ++j) {
            float4 a, b;
            entry_pair<WRAP_CUT>(list, j, a, b);
            const uint2 mk = masks[j];
            float2 dx = __fadd2_rn(make_float2(a.x, a.y), nx);
            float2 dy = __fadd2_rn(make_float2(a.z, a.w), ny);
            float2 dz = __fadd2_rn(make_float2(b.x, b.y), nz);
            if (WRAP_CUT) {
                dx = minus_image2(dx);
                dy = minus_image2(dy);
                dz = minus_image2(dz);
            }
            const float2 q = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, s2)));
            const bool u0 = (mk.x & lane_bit) != 0u, u1 = (mk.y & lane_bit) != 0u;
            const float2 w = make_float2(u0 && (!WRAP_CUT || q.x > cut) ? b.z : 0.f,
                                         u1 && (!WRAP_CUT || q.y > cut) ? b.w : 0.f);
            const float2 r = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
            const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(w, r), r), r);
            fx = __ffma2_rn(f, dx, fx);
            fy = __ffma2_rn(f, dy, fy);
            fz = __ffma2_rn(f, dz, fz);
        }
        ax[0] = fx.x; ax[1] = fx.y;
        ay[0] = fy.x; ay[1] = fy.y;
        az[0] = fz.x; az[1] = fz.y;
    } else {
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const float4 e = list[j];
            const bool u = (masks[j].x & lane_bit) != 0u;
#pragma unroll
            for (int b = 0; b < BPL; ++b) {
                float dx = e.x - x[b], dy = e.y - y[b], dz = e.z - z[b];
                if (WRAP_CUT) {
                    dx = minus_image(dx);
                    dy = minus_image(dy);
                    dz = minus_image(dz);
                }
                const float q = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, soft2)));
                const float r = rsqrt_normal(q);
                const float f = (u && (!WRAP_CUT || q > cut)) ? e.w * r * r * r : 0.f;
                ax[b] = fmaf(f, dx, ax[b]);
                ay[b] = fmaf(f, dy, ay[b]);
                az[b] = fmaf(f, dz, az[b]);
            }
        }
    }
}

// One per-body item for the lane's bodies: I = raw CoM and mass, J = (s,
// lo, hi, flags) with [lo, hi] the float32 band around s^2 / theta^2 where
// float64 decides, bodies in (m0, m1).  Adds the force of the bodies that
// accept; returns which of them open the node.
template <int BPL>
__device__ __forceinline__ void per_body_item(float4 I, float4 J, uint32_t m0, uint32_t m1, int lane,
                                              double th2d, float soft2, const float (&x)[BPL],
                                              const float (&y)[BPL], const float (&z)[BPL],
                                              float (&ax)[BPL], float (&ay)[BPL], float (&az)[BPL],
                                              bool (&opn)[BPL]) {
    const int flags = __float_as_int(J.w);
    if constexpr (BPL == 2) {
        float2 dx = __fadd2_rn(dup2(I.x), make_float2(-x[0], -x[1]));
        float2 dy = __fadd2_rn(dup2(I.y), make_float2(-y[0], -y[1]));
        float2 dz = __fadd2_rn(dup2(I.z), make_float2(-z[0], -z[1]));
        if (flags & kItemWrap) {
            dx = minus_image2(dx);
            dy = minus_image2(dy);
            dz = minus_image2(dz);
        }
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        bool a0 = d2.x > J.z, a1 = d2.y > J.z;
        const bool in0 = (m0 >> lane) & 1u, in1 = (m1 >> lane) & 1u;
        if (in0 && !a0 && !(d2.x < J.y)) a0 = ref_accepts_f64(J.x, th2d, dx.x, dy.x, dz.x);
        if (in1 && !a1 && !(d2.y < J.y)) a1 = ref_accepts_f64(J.x, th2d, dx.y, dy.y, dz.y);
        const bool u0 = in0 && a0, u1 = in1 && a1;
        opn[0] = in0 && !a0;
        opn[BPL - 1] = in1 && !a1;
        bool f0 = u0, f1 = u1;
        if (flags & kItemNear) {
            f0 = f0 && ref_outside_cut(dx.x, dy.x, dz.x, d2.x);
            f1 = f1 && ref_outside_cut(dx.y, dy.y, dz.y, d2.y);
        }
        // an item every reaching body opens adds no force (a third of them)
        if (!__any_sync(0xffffffffu, f0 || f1)) return;
        const float2 q = __fadd2_rn(d2, dup2(soft2));
        const float2 r = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
        const float2 w = make_float2(f0 ? I.w : 0.f, f1 ? I.w : 0.f);
        const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(w, r), r), r);
        const float2 fx = __ffma2_rn(f, dx, make_float2(ax[0], ax[1]));
        const float2 fy = __ffma2_rn(f, dy, make_float2(ay[0], ay[1]));
        const float2 fz = __ffma2_rn(f, dz, make_float2(az[0], az[1]));
        ax[0] = fx.x; ax[1] = fx.y;
        ay[0] = fy.x; ay[1] = fy.y;
        az[0] = fz.x; az[1] = fz.y;
    } else {
#pragma unroll
        for (int b = 0; b < BPL; ++b) {
            float dx = I.x - x[b], dy = I.y - y[b], dz = I.z - z[b];
            if (flags & kItemWrap) {
                dx = minus_image(dx);
                dy = minus_image(dy);
                dz = minus_image(dz);
            }
            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const bool in = ((b == 0 ? m0 : m1) >> lane) & 1u;
            bool a = d2 > J.z;
            if (in && !a && !(d2 < J.y)) a = ref_accepts_f64(J.x, th2d, dx, dy, dz);
            const bool u = in && a;
            opn[b] = in && !a;
            const bool fu = u && (!(flags & kItemNear) || ref_outside_cut(dx, dy, dz, d2));
            const float r = rsqrt_normal(d2 + soft2);
            const float f = fu ? I.w * r * r * r : 0.f;
            ax[b] = fmaf(f, dx, ax[b]);
            ay[b] = fmaf(f, dy, ay[b]);
            az[b] = fmaf(f, dz, az[b]);
        }
    }
}

// The rare outcome of a simple item: d^2 within the band around s^2 / theta^2.
// The reference's own float32 differences (from the node's record, not the
// shifted CoM of the item) and its float64 test.
static __device__ __noinline__ bool accepts_f64(const float4 *__restrict__ rec, int node, float box,
                                                double th2d, float x, float y, float z) {
    const float4 A = __ldg(rec + 2 * (int64_t)node);
    const float sx = __ldg(rec + 2 * (int64_t)node + 1).x;
    return ref_accepts_f64(sx > 0.5f * box ? box : sx, th2d, minus_image(A.x - x),
                           minus_image(A.y - y), minus_image(A.z - z));
}

// One simple item: its CoM at the one image every body of the bucket sees,
// out of the cut's reach.  For two bodies per lane I = (x, x, y, y), J = (z,
// z, m, node), K = (lo, hi, mask); for one I = (x, y, z, m), J.w = node.
// [lo, hi] is the band around s^2 / theta^2 where the float32 d^2 does not
// decide.  Adds the force of the bodies that accept the node and returns them
// (b0, b1): what is left of the mask opens it.
template <int BPL>
__device__ __forceinline__ uint2 simple_item(float4 I, float4 J, float4 K, uint32_t lane_bit,
                                             const float4 *rec, float box, double th2d, float soft2,
                                             const float (&x)[BPL], const float (&y)[BPL],
                                             const float (&z)[BPL], float (&ax)[BPL],
                                             float (&ay)[BPL], float (&az)[BPL]) {
    if constexpr (BPL == 2) {
        const float2 dx = __fadd2_rn(make_float2(I.x, I.y), make_float2(-x[0], -x[1]));
        const float2 dy = __fadd2_rn(make_float2(I.z, I.w), make_float2(-y[0], -y[1]));
        const float2 dz = __fadd2_rn(make_float2(J.x, J.y), make_float2(-z[0], -z[1]));
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        bool p0 = d2.x > K.y, p1 = d2.y > K.y;
        if ((!p0 && !(d2.x < K.x)) || (!p1 && !(d2.y < K.x))) {
            const int node = __float_as_int(J.w);
            if (!p0 && !(d2.x < K.x)) p0 = accepts_f64(rec, node, box, th2d, x[0], y[0], z[0]);
            if (!p1 && !(d2.y < K.x)) p1 = accepts_f64(rec, node, box, th2d, x[1], y[1], z[1]);
        }
        p0 = p0 && (__float_as_uint(K.z) & lane_bit) != 0u;
        p1 = p1 && (__float_as_uint(K.w) & lane_bit) != 0u;
        const uint2 acc = make_uint2(__ballot_sync(0xffffffffu, p0), __ballot_sync(0xffffffffu, p1));
        // an item every reaching body opens adds no force (a third of them)
        if ((acc.x | acc.y) == 0u) return acc;
        const float2 q = __fadd2_rn(d2, dup2(soft2));
        const float2 r = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
        const float2 w = make_float2(p0 ? J.z : 0.f, p1 ? J.z : 0.f);
        const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(w, r), r), r);
        const float2 fx = __ffma2_rn(f, dx, make_float2(ax[0], ax[1]));
        const float2 fy = __ffma2_rn(f, dy, make_float2(ay[0], ay[1]));
        const float2 fz = __ffma2_rn(f, dz, make_float2(az[0], az[1]));
        ax[0] = fx.x; ax[1] = fx.y;
        ay[0] = fy.x; ay[1] = fy.y;
        az[0] = fz.x; az[1] = fz.y;
        return acc;
    } else {
        const float dx = I.x - x[0], dy = I.y - y[0], dz = I.z - z[0];
        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        bool p = d2 > K.y;
        if (!p && !(d2 < K.x)) p = accepts_f64(rec, __float_as_int(J.w), box, th2d, x[0], y[0], z[0]);
        p = p && (__float_as_uint(K.z) & lane_bit) != 0u;
        const uint32_t acc = __ballot_sync(0xffffffffu, p);
        if (acc == 0u) return make_uint2(0u, 0u);
        const float r = rsqrt_normal(d2 + soft2);
        const float f = p ? I.w * r * r * r : 0.f;
        ax[0] = fmaf(f, dx, ax[0]);
        ay[0] = fmaf(f, dy, ay[0]);
        az[0] = fmaf(f, dz, az[0]);
        return make_uint2(acc, 0u);
    }
}

// Applies the first 32 entries of a list and moves the rest to the front.
// WRAP_CUT: the per-pair list (one float4 per entry), else the masked list.
template <int BPL, bool WRAP_CUT>
__device__ __forceinline__ void flush32(float4 *lst, uint2 *msk, int &cnt, int lane,
                                        const float (&x)[BPL], const float (&y)[BPL],
                                        const float (&z)[BPL], float soft2, float (&ax)[BPL],
                                        float (&ay)[BPL], float (&az)[BPL]) {
    constexpr int EW = WRAP_CUT ? 1 : entry_width<BPL>();
    apply_masked<BPL, WRAP_CUT>(lst, msk, 32, lane, x, y, z, soft2, ax, ay, az);
    __syncwarp();
#pragma unroll
    for (int w = 0; w < EW; ++w)
        if (lane < cnt - 32) lst[EW * lane + w] = lst[EW * (32 + lane) + w];
    if (lane < cnt - 32) msk[lane] = msk[32 + lane];
    cnt -= 32;
    __syncwarp();
}

// REDO false: the main pass over every bucket (work counter); true: the
// buckets a main pass with MAIN words gave up on (bucket record's fourth word =
// 1), found by a strided scan of the table and cleared when done.
// Twenty warps per SM with two bodies per lane, 28 with one (24 in blocks of
// eight).  Two bodies want their registers: bounded for 22 or 24 warps the
// kernel is 2 % faster to 6 % slower at 2M bodies and 8 to 13 % slower at 300k.
// One body leaves room: 128^3 one level 5.72 (16 warps) -> 4.88 ms (24).  The redo
// pass's region leaves ten warps their shared memory.
template <int BPL, int WARPS, int XW, bool REDO, bool TEST = false, int MAIN = XW>
__global__ void __launch_bounds__(WARPS * 32, (REDO ? 10 : BPL == 2 ? 20 : 28) / WARPS)
    k_forces_exact(GroupedParams P) {
    static_assert(BPL == 1 || BPL == 2, "one or two bodies per lane");
    extern __shared__ __align__(16) unsigned char x_smem[];
    constexpr int EW = entry_width<BPL>();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    float4 *f4 = reinterpret_cast<float4 *>(x_smem);
    float4 *mlist = f4 + wib * exact_f4_per_warp<BPL>();  // masked, one image, no cut
    float4 *xlist = mlist + kGList * EW;                  // per-pair image and cut, any mask
    float4 *plist = xlist + kGList;                       // per-body items (3 float4 each)
    uint2 *mbase = reinterpret_cast<uint2 *>(f4 + WARPS * exact_f4_per_warp<BPL>());
    uint2 *mmask = mbase + wib * kExactMasksPerWarp;
    uint2 *xmask = mmask + kGList;
    // the stack region: whole-bucket entries from word 0 up, (node, mask) entries from the end down
    int32_t *stack = reinterpret_cast<int32_t *>(mbase + WARPS * kExactMasksPerWarp) +
                     wib * XW;

    unsigned long long n_tests = 0, n_inter = 0, n_wrap = 0;
    int max_top = 0;
    bool overflow = false;
    const int n_buckets = P.ws[0];
    const float half_box = 0.5f * P.box;

    int4 *table = reinterpret_cast<int4 *>(P.ws + 4);  // the bucket records (P.buckets)
    // redo: this warp's share of the table, every `warps`-th record, 32 of them at a time (lane l
    // reads record chunk + l * warps: the records of a dense part of the system lie together);
    // marked holds those still to walk
    const int warps = gridDim.x * WARPS;
    int chunk = blockIdx.x * WARPS + wib;
    uint32_t marked = 0u;
    for (;;) {
        int g = 0;
        if (REDO) {
            while (marked == 0u && chunk < n_buckets) {
                const int r = chunk + lane * warps;
                marked = __ballot_sync(0xffffffffu, r < n_buckets && table[r].w == 1);
                if (marked == 0u) chunk += 32 * warps;
            }
            if (marked == 0u) break;
            g = chunk + (__ffs(marked) - 1) * warps;
            marked &= marked - 1u;
            if (marked == 0u) chunk += 32 * warps;
        } else {
            if (lane == 0) g = atomicAdd(P.ws + 1, 1);
            g = __shfl_sync(0xffffffffu, g, 0);
            if (g >= n_buckets) break;
            if (P.bucket_order) g = P.bucket_order[g];
        }
        const int4 bk = P.buckets[g];
        bool spill = false;  // main pass: this bucket is left to the redo pass
        uint32_t b_tests = 0, b_inter = 0, b_wrap = 0;  // this bucket's counts (lane's share)
        const int count = bk.y;
        float x[BPL], y[BPL], z[BPL];
        bool valid[BPL];
        float lx = INFINITY, ly = INFINITY, lz = INFINITY;
        float hx = -INFINITY, hy = -INFINITY, hz = -INFINITY;
#pragma unroll
        for (int b = 0; b < BPL; ++b) {
            const int k = lane + 32 * b;
            valid[b] = k < count;
            const int64_t i = (int64_t)bk.x + (valid[b] ? k : 0);
            x[b] = P.px[i];
            y[b] = P.py[i];
            z[b] = P.pz[i];
            if (valid[b]) {
                if (!(isfinite(x[b]) && isfinite(y[b]) && isfinite(z[b])))
                    set_flag(P.status, CNB_FLAG_NONFINITE);
                lx = fminf(lx, x[b]); ly = fminf(ly, y[b]); lz = fminf(lz, z[b]);
                hx = fmaxf(hx, x[b]); hy = fmaxf(hy, y[b]); hz = fmaxf(hz, z[b]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
            ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
            lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
            hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
            hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
            hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
        }
        const float gcx = 0.5f * (lx + hx), gcy = 0.5f * (ly + hy), gcz = 0.5f * (lz + hz);
        const float ghx = 0.5f * (hx - lx) + kBoxSlack, ghy = 0.5f * (hy - ly) + kBoxSlack,
                    ghz = 0.5f * (hz - lz) + kBoxSlack;
        // an entry whose image offset from the centre stays below this has one
        // minimum image for every body of the bucket
        const float wlx = 0.5f - ghx - 1e-6f, wly = 0.5f - ghy - 1e-6f, wlz = 0.5f - ghz - 1e-6f;
        // the bucket's bodies: bit l of word b is body l + 32 b
        const uint2 fm = make_uint2(count >= 32 ? 0xffffffffu : ((1u << count) - 1u),
                                    BPL == 1 || count <= 32 ? 0u
                                    : (count >= 64 ? 0xffffffffu : ((1u << (count - 32)) - 1u)));
        float th = P.theta, soft2 = P.soft2;
        double th2d = P.theta_sq;
        int32_t root = P.root;
        if (P.box_roots) {
            const uint64_t b = P.codes[bk.x] >> P.box_shift;
            const float4 bp = P.box_params[b];
            root = P.box_roots[b];
            th = bp.x;
            soft2 = bp.y * bp.y;
            th2d = (double)th * (double)th;
        }
        soft2 = normal_soft2(soft2);
        if (P.theta_per_bucket) {
            th = P.theta_per_bucket[g];
            th2d = (double)th * (double)th;
        }
        const float th2 = (float)th2d;
        const float inv_th2 = 1.f / th2;

        float ax[BPL], ay[BPL], az[BPL];
#pragma unroll
        for (int b = 0; b < BPL; ++b) ax[b] = ay[b] = az[b] = 0.f;
        int top = 1, ptop = 0, mcnt = 0, xcnt = 0, n_acc = 0;
        bool seeded = false;
        if (P.super_of_body) {
            const int sup = P.super_of_body[bk.x];
            const int4 h = sup >= 0 ? P.super_hdr[sup] : make_int4(0, 0, 0, 0);
            if (h.w && h.z <= XW) {
                // the nodes every body of the super-bucket accepts (k_super_lists)
                const float4 *far = P.far_lists + (int64_t)sup * P.far_cap;
                for (int j0 = 0; j0 < h.x; j0 += 32) {
                    const int c = min(32, h.x - j0);
                    if (lane < c) put_entry<BPL>(mlist, lane, far[j0 + lane]);
                    __syncwarp();
                    apply_entries<BPL, false, false>(mlist, c, x, y, z, soft2, ax, ay, az);
                    __syncwarp();
                }
                for (int j0 = 0; j0 < h.y; j0 += 32) {
                    const int c = min(32, h.y - j0);
                    if (lane < c) put_entry<BPL>(mlist, lane, far[P.far_cap - h.y + j0 + lane]);
                    __syncwarp();
                    apply_entries<BPL, true, true>(mlist, c, x, y, z, soft2, ax, ay, az);
                    __syncwarp();
                }
                if (lane == 0) {
                    b_inter += (uint32_t)((h.x + h.y) * count);
                    b_wrap += (uint32_t)(h.y * count);
                }
                const int32_t *near = P.near_lists + (int64_t)sup * P.near_cap;
                for (int j = lane; j < h.z; j += 32) stack[j] = near[j];
                top = h.z;
                seeded = true;
            }
        }
        if (!seeded && lane == 0) stack[0] = root;
        __syncwarp();
        uint32_t rounds = 0;
        int narrow = 0;     // rounds of fewer than kXLeast entries
        bool wide = false;  // redo: the main pass has given up here
        while ((top > 0 || ptop > 0) && !spill) {
            // a valid tree pushes every node at most once per bucket
            if (++rounds > (uint32_t)P.m_nodes) {
                if (lane == 0) set_flag(P.status, CNB_FLAG_BAD_TOPOLOGY);
                break;
            }
            // A popped entry leaves at most five words more than it took (a whole-bucket entry
            // opened by part of the bucket: one word becomes two (node, mask) entries), so
            // popping a fifth of the free words never overflows the region.
            // The redo pass goes by the main pass's region (MAIN) for as long as that lasts: the
            // same order of nodes, so the same sums.
            const int used = top + 3 * ptop;
            int room = ((MAIN - used) * 51) >> 8;
            if (room < kXLeast && !(REDO && wide)) {
                if (room <= 0 || ++narrow > kXNarrow) {
                    if (!REDO) {
                        spill = true;
                        break;
                    }
                    wide = true;
                }
            }
            if (REDO && wide) {
                if (used + 5 > XW) {
                    overflow = spill = true;
                    break;
                }
                room = max(((XW - kXDeep - used) * 51) >> 8, 1);
            }
            // part-bucket entries first (they keep the second stack short)
            const int k1 = min(ptop, min(32, room));
            const int k2 = min(top, min(32, room) - k1);
            ptop -= k1;
            top -= k2;
            int32_t node = -1;
            uint2 mk = fm;
            if (lane < k1) {
                const int pw = part_word<XW>(ptop + lane);
                node = stack[pw];
                mk = make_uint2((uint32_t)stack[pw + 1], (uint32_t)stack[pw + 2]);
            } else if (lane < k1 + k2) {
                node = stack[top + lane - k1];
            }
            __syncwarp();
            if (node >= P.m_nodes) {
                set_flag(P.status, CNB_FLAG_BAD_TOPOLOGY);
                node = -1;
            }
            // 1: accepted by every body of the mask, 2: opened by every one, 3: per body
            int cls = 0;
            bool one_image = false, simple = false, shifted = false, near_box = false;
            float4 A = make_float4(0.f, 0.f, 0.f, 0.f), E = A;
            float s = 0.f;
            int32_t c0 = -1, c1 = -1;
            if (node >= 0) {
                A = __ldg(P.rec + 2 * node);
                const float4 S = __ldg(P.rec + 2 * node + 1);
                if (A.w > 0.f) {  // physics_kernels.py:114 (nm <= 0: skipped)
                    c0 = __float_as_int(S.z);
                    c1 = __float_as_int(S.w);
                    const float dx = A.x - gcx, dy = A.y - gcy, dz = A.z - gcz;
                    const float sx_ = image_of(dx), sy_ = image_of(dy), sz_ = image_of(dz);
                    const float adx = fabsf(dx - sx_), ady = fabsf(dy - sy_), adz = fabsf(dz - sz_);
                    const float tx = fmaxf(adx - ghx, 0.f), ty = fmaxf(ady - ghy, 0.f),
                                tz = fmaxf(adz - ghz, 0.f);
                    const float d2min = tx * tx + ty * ty + tz * tz;
                    s = S.x > half_box ? P.box : S.x;  // physics_kernels.py:131-132
                    if (c0 == -1) {
                        cls = 1;  // a leaf: used by every body that reaches it
                    } else {
                        const float ux = fminf(adx + ghx, half_box), uy = fminf(ady + ghy, half_box),
                                    uz = fminf(adz + ghz, half_box);
                        const float d2max = ux * ux + uy * uy + uz * uz;
                        const float s2 = s * s;
                        if (s2 < th2 * d2min * (1.f - kRelMargin)) cls = 1;
                        else if (s2 > th2 * d2max * (1.f + kRelMargin)) cls = 2;
                        else cls = 3;
                    }
                    near_box = d2min <= kCutGuard;
                    one_image = adx < wlx && ady < wly && adz < wlz;
                    shifted = sx_ != 0.f || sy_ != 0.f || sz_ != 0.f;
                    E = make_float4(A.x - sx_, A.y - sy_, A.z - sz_, A.w);
                    // a per-body item takes the shifted CoM when the shift is exact in float32
                    simple = one_image && !near_box && E.x + sx_ == A.x && E.y + sy_ == A.y &&
                             E.z + sz_ == A.z;
                }
            }
            b_tests += (node >= 0);
            const bool to_m = cls == 1 && one_image && !near_box;
            const bool to_x = cls == 1 && !(one_image && !near_box);
            const uint32_t m_msk = __ballot_sync(0xffffffffu, to_m);
            const uint32_t m_x = __ballot_sync(0xffffffffu, to_x);
            const uint32_t m_ps = __ballot_sync(0xffffffffu, cls == 3 && simple);
            const uint32_t m_pg = __ballot_sync(0xffffffffu, cls == 3 && !simple);
            if (cls == 1) {
                const int nb = __popc(mk.x) + __popc(mk.y);
                b_inter += nb;
                if (to_m) {
                    const int w = mcnt + __popc(m_msk & lt);
                    put_entry<BPL>(mlist, w, E);
                    mmask[w] = mk;
                } else {
                    const int w = xcnt + __popc(m_x & lt);
                    xlist[w] = A;
                    xmask[w] = mk;
                    b_wrap += nb;
                }
            }
            mcnt += __popc(m_msk);
            xcnt += __popc(m_x);
            // per-body items: the simple ones from the front of the list, the others (per-pair
            // image or cut) from its end; lane l remembers the slot of its own
            const int n_ps = __popc(m_ps), n_pg = __popc(m_pg);
            int slot = -1;
            if (cls == 3) {
                // the band [lo, hi] around s^2 / theta^2 inside which float64 decides.  A shifted
                // CoM gives differences within 2^-25 + 2^-26 of the reference's, d^2 within
                // 2 sqrt(3) d of that: 3e-7 d covers it twice.
                const float R = s * s * inv_th2;
                const float widen = simple && shifted ? 3e-7f * sqrtf(R) : 0.f;
                const float lo = R * (1.f - kRelMargin) - widen, hi = R * (1.f + kRelMargin) + widen;
                const float m0 = __uint_as_float(mk.x), m1 = __uint_as_float(mk.y);
                slot = simple ? __popc(m_ps & lt) : 31 - __popc(m_pg & lt);
                float4 *item = plist + 3 * slot;
                if (simple) {
                    if (BPL == 2) {
                        item[0] = make_float4(E.x, E.x, E.y, E.y);
                        item[1] = make_float4(E.z, E.z, E.w, __int_as_float(node));
                    } else {
                        item[0] = E;
                        item[1] = make_float4(0.f, 0.f, 0.f, __int_as_float(node));
                    }
                    item[2] = make_float4(lo, hi, m0, m1);
                } else {
                    const int fl = (one_image && !shifted ? 0 : kItemWrap) | (near_box ? kItemNear : 0);
                    item[0] = A;
                    item[1] = make_float4(s, lo, hi, __int_as_float(fl));
                    item[2] = make_float4(0.f, 0.f, m0, m1);
                }
            }
            __syncwarp();
            // every body of the mask decides for itself; a lane keeps the mask of the bodies that
            // accept its own item, and the children of the items that some body opened are pushed
            // together afterwards
            uint2 my_acc = make_uint2(0u, 0u);
#pragma unroll 1
            for (int j = 0; j < n_ps; ++j) {
                const uint2 acc = simple_item<BPL>(plist[3 * j], plist[3 * j + 1], plist[3 * j + 2],
                                                   1u << lane, P.rec, P.box, th2d, soft2, x, y, z, ax,
                                                   ay, az);
                if (lane == 0) *reinterpret_cast<uint2 *>(plist + 3 * j + 2) = acc;
            }
#pragma unroll 1
            for (int j = 31; j > 31 - n_pg; --j) {
                const float4 K = plist[3 * j + 2];
                bool opn[BPL];
                per_body_item<BPL>(plist[3 * j], plist[3 * j + 1], __float_as_uint(K.z),
                                   __float_as_uint(K.w), lane, th2d, soft2, x, y, z, ax, ay, az, opn);
                const uint32_t o0 = __ballot_sync(0xffffffffu, opn[0]);
                const uint32_t o1 = BPL == 2 ? __ballot_sync(0xffffffffu, opn[BPL - 1]) : 0u;
                if (lane == 0) *reinterpret_cast<uint2 *>(plist + 3 * j + 2) = make_uint2(~o0, ~o1);
            }
            __syncwarp();
            if (cls == 3) my_acc = *reinterpret_cast<uint2 *>(plist + 3 * slot + 2);
            {
                // the bodies of each node's mask that open it: all, or those that did not accept
                uint2 my_om = make_uint2(0u, 0u);
                if (cls == 2) my_om = mk;
                if (cls == 3) {
                    my_om = make_uint2(mk.x & ~my_acc.x, mk.y & ~my_acc.y);
                    n_acc += __popc(mk.x & my_acc.x) + __popc(mk.y & my_acc.y);
                }
                const bool has = (my_om.x | my_om.y) != 0u;
                const bool whole_o = my_om.x == fm.x && my_om.y == fm.y;
                const uint32_t mw = __ballot_sync(0xffffffffu, has && whole_o);
                const uint32_t mp = __ballot_sync(0xffffffffu, has && !whole_o);
                const int nw = __popc(mw), npart = __popc(mp);
                {
                    if (has && whole_o) {
                        const int pos = top + 2 * __popc(mw & lt);
                        stack[pos] = c1;
                        stack[pos + 1] = c0;
                    }
                    if (has && !whole_o) {
                        const int pos = ptop + 2 * __popc(mp & lt);
                        const int w1 = part_word<XW>(pos), w0 = part_word<XW>(pos + 1);
                        stack[w1] = c1;
                        stack[w1 + 1] = (int32_t)my_om.x;
                        stack[w1 + 2] = (int32_t)my_om.y;
                        stack[w0] = c0;
                        stack[w0 + 1] = (int32_t)my_om.x;
                        stack[w0 + 2] = (int32_t)my_om.y;
                    }
                    top += 2 * nw;
                    ptop += 2 * npart;
                }
            }
            max_top = max(max_top, top + 3 * ptop);  // words of the stack region
            __syncwarp();
            if (mcnt >= 32) flush32<BPL, false>(mlist, mmask, mcnt, lane, x, y, z, soft2, ax, ay, az);
            if (xcnt >= 32) flush32<BPL, true>(xlist, xmask, xcnt, lane, x, y, z, soft2, ax, ay, az);
            // tests: give up on a bucket after its first round as an overflow would
            if (TEST && rounds == 1 && g % P.test_spill_every == 0) spill = true;
        }
        if (!REDO && spill) {
            // given up: no force and no counts from this pass; the redo
            // pass walks it again
            if (lane == 0) table[g].w = 1;
            __syncwarp();
            continue;
        }
        apply_masked<BPL, false>(mlist, mmask, mcnt, lane, x, y, z, soft2, ax, ay, az);
        apply_masked<BPL, true>(xlist, xmask, xcnt, lane, x, y, z, soft2, ax, ay, az);
        __syncwarp();
        if (REDO && lane == 0) table[g].w = 0;
        n_tests += b_tests;
        n_inter += b_inter + n_acc;
        n_wrap += b_wrap + n_acc;
#pragma unroll
        for (int b = 0; b < BPL; ++b) {
            if (valid[b]) {
                const int64_t i = (int64_t)bk.x + lane + 32 * b;
                const float fx = P.G * ax[b], fy = P.G * ay[b], fz = P.G * az[b];
                P.force[3 * i] = fx;
                P.force[3 * i + 1] = fy;
                P.force[3 * i + 2] = fz;
                if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz))
                    set_flag(P.status, CNB_FLAG_NONFINITE);
            }
        }
    }
    if (overflow && lane == 0) set_flag(P.status, CNB_FLAG_LIST_OVERFLOW);
    if (P.stats) {
        for (int o = 16; o > 0; o >>= 1) {
            n_tests += __shfl_xor_sync(0xffffffffu, n_tests, o);
            n_inter += __shfl_xor_sync(0xffffffffu, n_inter, o);
            n_wrap += __shfl_xor_sync(0xffffffffu, n_wrap, o);
        }
        if (lane == 0) {
            atomicAdd(P.stats, n_inter);
            atomicAdd(P.stats + 1, n_tests);
            atomicAdd(P.stats + 2, n_wrap);
        }
    }
    if (lane == 0) atomicMax(P.ws + 2, max_top);
}

template <int BPL, int WARPS, int XW, bool REDO, bool TEST = false, int MAIN = XW>
static int launch_exact_pass(GroupedParams &P, cudaStream_t st) {
    const size_t smem = exact_smem<BPL>(WARPS, XW);
    const auto kernel = k_forces_exact<BPL, WARPS, XW, REDO, TEST, MAIN>;
    CNB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, WARPS * 32, smem);
    // persistent grid: the work counter (main pass) or the table scan (redo) hands out buckets
    kernel<<<kSMs * (per_sm > 0 ? per_sm : 1), WARPS * 32, smem, st>>>(P);
    return launch_status();
}

template <int BPL, int WARPS, int MAIN>
static int launch_exact_region(GroupedParams &P, cudaStream_t st) {
    if (P.test_spill_every > 0)  // tests: the main pass gives up on every n-th bucket
        CNB_TRY((launch_exact_pass<BPL, WARPS, MAIN, false, true>(P, st)));
    else
        CNB_TRY((launch_exact_pass<BPL, WARPS, MAIN, false>(P, st)));
    // the buckets it gave up on, if any (otherwise every warp scans its share of the
    // bucket table and returns)
    return launch_exact_pass<BPL, 2, kXWordsRedo, true, false, MAIN>(P, st);
}

template <int BPL, int WARPS>
static int launch_exact_shape(GroupedParams &P, cudaStream_t st) {
    if (P.box_roots) return launch_exact_region<BPL, WARPS, kXWords>(P, st);
    if (P.theta < 0.25f) return launch_exact_region<BPL, WARPS, kXWordsWidest>(P, st);
    if (P.theta < 0.4f) return launch_exact_region<BPL, WARPS, kXWordsWide>(P, st);
    return launch_exact_region<BPL, WARPS, BPL == 2 ? kXWordsTwo : kXWords>(P, st);
}

static int g_test_spill_every = 0;  // cnb_exact_test_spill

// Systems of at most CNB_EXACT_WALK_BODIES bodies take the walk by groups
// (forces_ref.cu), super-buckets or not: their few hundred buckets leave most
// warps of the chip idle while each is a serial walk of some 80 000 instructions.  Measured on even and clustered states at theta 0.4, 0.5,
// 0.7 and 0.9 (us at 0.5, the fastest of six bucket shapes, one and two levels /
// groups; in brackets the geometric mean over all states and angles of groups
// against buckets): 20 000 bodies 162 and 184 / 80 and 90 (0.50), 50 000 226 and
// 258 / 184 and 207 (0.79), 65 536 229 and 285 / 238 and 262 (0.96), 80 000 264 and
// 365 / 283 and 315 (0.94), 98 304 342 and 401 / 365 and 391 (1.00), 131 072 377 and
// 478 / 487 and 526 (1.15).  Even states at small angles cross earlier (0.4: between
// 50 000 and 65 536), clustered ones and large angles later; below theta 0.4 the
// groups need a larger stack and the line is CNB_EXACT_WALK_BODIES_SMALL_ANGLE (see
// forces_ref.cu).
int launch_exact(GroupedParams &P, int bodies_per_lane, int block_warps, cudaStream_t st) {
    const int64_t groups = P.theta < 0.4f ? CNB_EXACT_WALK_BODIES_SMALL_ANGLE : CNB_EXACT_WALK_BODIES;
    if (P.n <= groups && !P.box_roots && !P.theta_per_bucket) return launch_exact_walk(P, st);
    P.test_spill_every = g_test_spill_every;
    switch (bodies_per_lane * 16 + block_warps) {
        case 16 + 2: return launch_exact_shape<1, 2>(P, st);
        case 16 + 4: return launch_exact_shape<1, 4>(P, st);
        case 16 + 8: return launch_exact_shape<1, 8>(P, st);
        case 32 + 2: return launch_exact_shape<2, 2>(P, st);
        case 32 + 4: return launch_exact_shape<2, 4>(P, st);
        case 32 + 8: return launch_exact_shape<2, 8>(P, st);
        default: return CNB_E_INVALID_ARG;
    }
}

}  // namespace cnb

extern "C" int cnb_exact_test_spill(int every) {
    if (every < 0) return CNB_E_INVALID_ARG;
    cnb::g_test_spill_every = every;
    return CNB_OK;
}
