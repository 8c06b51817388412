// sort_persistent.cu -- the stable LSD radix sort of (key, index) pairs as one
// launch (src/core/state.py:35 `cp.argsort(codes)`).
//
// The one-sweep sort (sort.cu) is ten launches, each a chain of load, rank,
// look-back and scatter that a small sort mostly waits in and a large one
// spends polling the tiles before it.  Here one block per SM stays for all
// passes, with a contiguous chunk of at most 14 336 keys that it holds in
// registers.  A pass is
//   rank     stable ranks in the chunk (a ballot per digit bit finds the lanes
//            of a digit, per-warp counters give the order)
//   publish  the chunk's 256 digit counts; grid barrier
//   place    the counts of the blocks before it and of all blocks are added up
//            from the published rows, the chunk is put in digit order in shared
//            memory and written out in runs; grid barrier
//
// The barriers need all blocks resident: a cooperative launch.  Their waits
// are bounded (CNB_FLAG_WAIT_LIMIT, as the one-sweep sort's).  Data other
// blocks wrote is read through L2 (__ldcg): the buffers are reused.
//
// Measured on 63-bit keys, one-sweep against this (us): 4096 keys 104 / 58,
// 65 536 118 / 73, 1 000 003 202 / 150, 2 097 152 347 / 236.  More keys would
// need a second chunk per block, read twice: 2.1M 305, 16.8M 2076 against 1647
// of the one-sweep launches with ballots, which those sizes keep.
#include "ctx.cuh"

namespace cnb {

namespace {

constexpr int kPThreads = 1024;
constexpr int kPWarps = kPThreads / 32;
constexpr int kPParts = kPThreads / 256;  // threads per digit
// keys per thread: 8 while one block per SM holds all keys so (1.2M on 148 SMs), 14 up to 2.1M
// (64 registers: the keys of a chunk and their ranks; 12 spilt words at 14)
constexpr int kPItems = 8, kPItemsMost = 14;
constexpr int persistent_smem(int items) {
    return kPThreads * items * (int)(sizeof(uint64_t) + sizeof(uint32_t)) + kPWarps * 256 * 4;
}

struct PersistentSort {
    const uint64_t *kin;
    const uint32_t *vin;  // null: identity
    uint64_t *kout;
    uint32_t *vout;
    uint64_t *ktmp[2];
    uint32_t *vtmp[2];
    int64_t n, chunk;  // chunk: keys per block, a multiple of kPThreads
    int passes;
    uint32_t *hist;  // [blocks][256]
    uint32_t *bar;   // arrivals; zero at launch
    int32_t *flags;
    const int32_t *skip;
    unsigned long long *stat;
    int wait_limit;
    int withheld;  // tests: the block that never arrives (-1: none)
};

// Waits until every block has arrived `target` / gridDim.x times; false when
// the wait gave up.  Orders all of the block's earlier writes before all of
// the other blocks' later reads.
__device__ __forceinline__ bool grid_wait(const PersistentSort &P, uint32_t target, int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = (int)blockIdx.x != P.withheld;
        __threadfence();
        if (ok) atomicAdd(P.bar, 1u);
        int spins = 0;
        while (ok && *(volatile uint32_t *)P.bar < target) {
            if (++spins > P.wait_limit) {
                set_flag(P.flags, CNB_FLAG_WAIT_LIMIT);
                ok = 0;
                break;
            }
            if (spins > 64) __nanosleep(32);
        }
        __threadfence();
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// Exclusive scan of one value per digit thread (threads 0..255); ws: 8 words.
__device__ __forceinline__ uint32_t digit_exscan(uint32_t v, uint32_t *ws) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (warp < 8 && lane == 31) ws[warp] = incl;
    __syncthreads();
    uint32_t base = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) base += (w < warp) ? ws[w] : 0u;
    __syncthreads();
    return base + incl - v;
}

// Stable rank of every key among its warp's keys of the same digit; the
// warp's digit counts are left in wcnt (zero on entry).  left: the keys from
// the warp's first one to the end of the chunk.
template <int ITEMS>
__device__ __forceinline__ void rank_keys(const uint64_t (&key)[ITEMS], uint32_t (&rank)[ITEMS],
                                          uint32_t *wcnt, int shift, int64_t left, int items) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        if (r >= items || left <= r * 32) break;
        const int64_t row = left - r * 32;  // keys of this row
        const uint32_t d = (uint32_t)(key[r] >> shift) & 255u;
        const bool valid = lane < row;
        uint32_t m = row >= 32 ? 0xffffffffu : (1u << row) - 1u;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1u;
            const uint32_t v = __ballot_sync(0xffffffffu, bit);
            m &= bit ? v : ~v;
        }
        const uint32_t before = valid ? wcnt[d] : 0u;
        __syncwarp();
        if (valid && (m & lt) == 0u) wcnt[d] = before + __popc(m);
        __syncwarp();
        rank[r] = before + __popc(m & lt);
    }
}

template <int ITEMS>
__global__ void __launch_bounds__(kPThreads, 1) k_sort_persistent(PersistentSort P) {
    if (P.skip && *(volatile const int32_t *)P.skip) return;
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *skey = reinterpret_cast<uint64_t *>(smem);
    uint32_t *sval = reinterpret_cast<uint32_t *>(skey + kPThreads * ITEMS);
    uint32_t *wcnt = sval + kPThreads * ITEMS;  // [warps][256]
    __shared__ uint32_t s_part[kPParts][256], s_tot[kPParts][256];
    __shared__ uint32_t gbase[256], tstart[256], ws[8];
    __shared__ int s_ok;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int dg = threadIdx.x & 255, part = threadIdx.x >> 8;
    const int items = (int)(P.chunk / kPThreads);
    const int64_t lo = blockIdx.x * P.chunk, hi = min(P.n, lo + P.chunk);
    const int64_t wb = lo + (int64_t)warp * 32 * items;  // this warp's keys: wb + r * 32 + lane
    const int blocks = gridDim.x;
    uint32_t arrivals = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0 && P.stat) atomicAdd(P.stat, 1ull);

    const uint64_t *ks = P.kin;
    const uint32_t *vs = P.vin;
    for (int p = 0; p < P.passes; ++p) {
        const bool last = p == P.passes - 1;
        uint64_t *kd = last ? P.kout : P.ktmp[p & 1];
        uint32_t *vd = last ? P.vout : P.vtmp[p & 1];
        const int shift = 8 * p;
        uint64_t key[ITEMS];
        uint32_t rank[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int64_t e = wb + r * 32 + lane;
            key[r] = r < items && e < hi ? __ldcg(ks + e) : 0;
        }
        for (int i = threadIdx.x; i < kPWarps * 256; i += kPThreads) wcnt[i] = 0u;
        __syncthreads();
        rank_keys(key, rank, wcnt + warp * 256, shift, hi - wb, items);
        __syncthreads();
        // the chunk's digit counts, and in wcnt where a warp's keys of a digit start among them
        uint32_t count = 0;
        {
            constexpr int kEach = kPWarps / kPParts;
            uint32_t c[kEach], sum = 0;
#pragma unroll
            for (int k = 0; k < kEach; ++k) {
                c[k] = wcnt[(part * kEach + k) * 256 + dg];
                sum += c[k];
            }
            s_part[part][dg] = sum;
            __syncthreads();
            uint32_t run = 0;
#pragma unroll
            for (int q = 0; q < kPParts; ++q) {
                run += q < part ? s_part[q][dg] : 0u;
                count += s_part[q][dg];
            }
#pragma unroll
            for (int k = 0; k < kEach; ++k) {
                wcnt[(part * kEach + k) * 256 + dg] = run;
                run += c[k];
            }
        }
        uint32_t before = 0, all = count;
        if (blocks > 1) {
            if (part == 0) __stcg(P.hist + (int64_t)blockIdx.x * 256 + dg, count);
            arrivals += blocks;
            if (!grid_wait(P, arrivals, &s_ok)) return;
            // a quarter of the blocks' rows per thread
            const int q = (blocks + kPParts - 1) / kPParts;
            const int b0 = part * q, b1 = min(blocks, b0 + q);
            uint32_t bef = 0, tot = 0;
#pragma unroll 8
            for (int b = b0; b < b1; ++b) {
                const uint32_t v = __ldcg(P.hist + (int64_t)b * 256 + dg);
                tot += v;
                bef += b < (int)blockIdx.x ? v : 0u;
            }
            s_part[part][dg] = bef;
            s_tot[part][dg] = tot;
            __syncthreads();
            all = 0;
#pragma unroll
            for (int k = 0; k < kPParts; ++k) {
                before += s_part[k][dg];
                all += s_tot[k][dg];
            }
        }
        const uint32_t start = digit_exscan(part == 0 ? all : 0u, ws);
        if (part == 0) gbase[dg] = start + before;
        const uint32_t ts = digit_exscan(part == 0 ? count : 0u, ws);
        if (part == 0) tstart[dg] = ts;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int64_t e = wb + r * 32 + lane;
            if (r < items && e < hi) {
                const uint32_t d = (uint32_t)(key[r] >> shift) & 255u;
                const uint32_t at = tstart[d] + wcnt[warp * 256 + d] + rank[r];
                skey[at] = key[r];
                sval[at] = vs ? __ldcg(vs + e) : (uint32_t)e;
            }
        }
        __syncthreads();
        const int tile_n = (int)(hi - lo);
        for (int j = threadIdx.x; j < tile_n; j += kPThreads) {
            const uint64_t k = skey[j];
            const uint32_t d = (uint32_t)(k >> shift) & 255u;
            const int64_t at = (int64_t)gbase[d] + (j - tstart[d]);
            kd[at] = k;
            vd[at] = sval[j];
        }
        ks = kd;
        vs = vd;
        if (!last) {
            arrivals += blocks;
            if (blocks == 1) {
                __threadfence_block();
                __syncthreads();
            } else if (!grid_wait(P, arrivals, &s_ok)) {
                return;
            }
        }
    }
}

}  // namespace

// The blocks of the persistent sort that can be resident together on the
// current device (0: no cooperative launches, or it does not fit).
int persistent_blocks() {
    int dev = 0, coop = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || !coop) {
        cudaGetLastError();
        return 0;
    }
    const auto fits = [](const void *f, int smem) {
        int b = 0;
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
               cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kPThreads, smem) == cudaSuccess && b > 0;
    };
    if (!fits((const void *)k_sort_persistent<kPItems>, persistent_smem(kPItems)) ||
        !fits((const void *)k_sort_persistent<kPItemsMost>, persistent_smem(kPItemsMost))) {
        cudaGetLastError();
        return 0;
    }
    return sms;
}

// The most keys it takes on this context: one register-resident chunk per block.
int64_t persistent_max(const cnb_ctx *ctx) {
    return (int64_t)ctx->persistent_blocks * kPThreads * kPItemsMost;
}

int sort_pairs_persistent(cnb_ctx *ctx, const uint64_t *keys_in, uint64_t *keys_out,
                          const uint32_t *idx_in, uint32_t *perm_out, int64_t n, int key_bits,
                          cudaStream_t st, const int32_t *skip, uint32_t *arrivals) {
    PersistentSort P{};
    P.passes = (key_bits + 7) / 8;
    if (P.passes == 1 && (keys_in == keys_out || (idx_in && idx_in == perm_out))) P.passes = 2;
    P.kin = keys_in;
    P.vin = idx_in;
    P.kout = keys_out;
    P.vout = perm_out;
    for (int k = 0; k < 2; ++k) {
        P.ktmp[k] = ctx->keys_tmp[k];
        P.vtmp[k] = ctx->vals_tmp[k];
    }
    P.n = n;
    // one block up to 8 K keys (no barrier); then a block per 1024 keys until every SM has one
    const int64_t per = n <= 8 * kPThreads ? n : (n + ctx->persistent_blocks - 1) / ctx->persistent_blocks;
    P.chunk = (per + kPThreads - 1) / kPThreads * kPThreads;
    const int blocks = (int)((n + P.chunk - 1) / P.chunk);
    // the one-sweep sort's scratch: the arrivals in its first word, the rows behind its counters
    P.bar = arrivals ? arrivals : ctx->sweep;
    P.hist = ctx->sweep + kSweepMetaWords;
    P.flags = ctx->flags;
    P.skip = skip;
    P.stat = ctx->sort_stats ? ctx->sort_stats + 1 : nullptr;
    P.wait_limit = ctx->barrier_wait_limit > 0 ? ctx->barrier_wait_limit : 1 << 22;
    P.withheld = ctx->withheld_block;
    if (!arrivals && blocks > 1) CNB_CUDA(cudaMemsetAsync(P.bar, 0, sizeof(uint32_t), st));
    void *args[] = {&P};
    const bool few = P.chunk <= kPThreads * kPItems;
    const cudaError_t e = cudaLaunchCooperativeKernel(
        few ? (const void *)k_sort_persistent<kPItems> : (const void *)k_sort_persistent<kPItemsMost>,
        dim3((unsigned)blocks), dim3(kPThreads), args, persistent_smem(few ? kPItems : kPItemsMost), st);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kNotResident;
    }
    CNB_CUDA(e);
    return launch_status();
}

}  // namespace cnb
