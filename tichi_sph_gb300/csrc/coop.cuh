// Pieces of the cooperative kernels: the grid-wide barrier, each block's share of the
// items, sums in the order of the separate kernels, the launch.
#pragma once

#include <type_traits>
#include <utility>

#include "ctx.h"

namespace tsph {

// A poll of the barrier's counter takes about half a microsecond: the limit is
// a few seconds, after which the step is given up and the next reading of the
// scalars says so.
constexpr unsigned int kSpinLimit = 1u << 23;

// Barrier over the grid's blocks (all resident: a cooperative launch).  The
// counter only grows within a launch; the launch's last block to leave sets it
// back.  False: a block did not arrive within the limit; every block then leaves.
struct GridBarrier {
    unsigned int *bar;  // words kBarCount, kBarGaveUp, kBarLeft
    // the count to wait for; starts at the blocks that will not come (0 but in tests,
    // tsph_set_absent_blocks), for which the wait is a short one
    unsigned int target;
    static __device__ __forceinline__ unsigned int acquire(const unsigned int *p) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ bool sync() {
        __shared__ int ok;
        __syncthreads();
        if (threadIdx.x == 0) {
            target += gridDim.x;
            // release / acquire at GPU scope, with the block's two barriers around
            // them, order everything before against everything after
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar + kBarCount) : "memory");
            bool all = true;
            unsigned int n = 0;
            while (acquire(bar + kBarCount) < target) {
                if ((++n & 1023u) != 0) continue;
                if (n > kSpinLimit || target % gridDim.x != 0) atomicExch(bar + kBarGaveUp, 1u);
                if (acquire(bar + kBarGaveUp)) {
                    all = false;
                    break;
                }
            }
            ok = all;
        }
        __syncthreads();
        return ok != 0;
    }
};

// The block's share of n items: contiguous runs of 32, shares that differ by one
// run at most.
struct WarpShare {
    unsigned int first, runs;
    __device__ __forceinline__ WarpShare(int64_t n) {
        const unsigned int nw = (unsigned int)((n + 31) >> 5), per = nw / gridDim.x, more = nw % gridDim.x;
        first = blockIdx.x * per + min(blockIdx.x, more);
        runs = per + (blockIdx.x < more ? 1u : 0u);
    }
    __device__ __forceinline__ unsigned int run(unsigned int w) const { return first + w; }
};

// The block's share of n items where its warps take several runs each (QUEUE): up to
// kDealt runs per block WarpShare's, whose neighbours share the SM's L1, from
// there on groups of 16 neighbouring runs dealt to the blocks in turn.  Once a
// flow has developed, a share that lies together is all surface or all interior, and
// a sweep waits for the interior's (us a substep of a dam break after 500
// substeps, together and dealt: 439k 706 / 716, 512k 849 / 809, 1M
// 1535 / 1385; with groups of 8 the 1M step from rest takes 5% longer).
struct QueueShare {
    static constexpr unsigned int kGroup = 16, kDealt = 96;
    unsigned int first, runs, skip;  // skip: runs between the block's groups
    __device__ __forceinline__ QueueShare(int64_t n) {
        const unsigned int nw = (unsigned int)((n + 31) >> 5);
        if (nw >= kDealt * gridDim.x) {
            const unsigned int ng = (nw + kGroup - 1) / kGroup, per = ng / gridDim.x, more = ng % gridDim.x;
            first = blockIdx.x * kGroup;
            runs = (per + (blockIdx.x < more ? 1u : 0u)) * kGroup;
            if ((ng - 1) % gridDim.x == blockIdx.x) runs -= ng * kGroup - nw;
            skip = (gridDim.x - 1) * kGroup;
        } else {
            const WarpShare w(n);
            first = w.first;
            runs = w.runs;
            skip = 0;
        }
    }
    // the block's w-th run
    __device__ __forceinline__ unsigned int run(unsigned int w) const { return first + w + w / kGroup * skip; }
};

// What a block's warps take runs from: a count in shared memory, and its value at
// the start of the phase (the same in every thread).
struct RunQueue {
    unsigned int *next;
    unsigned int base;
};

// Runs ff(i, run) over the fluid's nf items and fb(i) over the boundary's nb in
// the block's warps (every lane of a warp calls, i may be past the end).  With QUEUE
// a warp takes its first run by its place and the others as it gets to them; two
// calls are then a barrier of the block apart.
template <bool QUEUE, class FF, class FB>
__device__ __forceinline__ void for_items(RunQueue &q, int64_t nf, int64_t nb, FF &&ff, FB &&fb) {
    using Share = std::conditional_t<QUEUE, QueueShare, WarpShare>;
    const Share f(nf), b(nb);
    const int lane = threadIdx.x & 31;
    const unsigned int warps = blockDim.x >> 5, total = f.runs + b.runs;
    for (unsigned int w = threadIdx.x >> 5; w < total;) {
        if (w < f.runs) {
            const int64_t r = f.run(w);
            ff(r * 32 + lane, r);
        } else {
            fb((int64_t)b.run(w - f.runs) * 32 + lane);
        }
        if (!QUEUE) {
            w += warps;
        } else {
            if (total <= warps) break;
            if (lane == 0) w = warps + (atomicAdd(q.next, 1u) - q.base);
            w = __shfl_sync(0xffffffffu, w, 0);
        }
    }
    // (total - warps taken, and every warp once more in vain)
    if (QUEUE && total > warps) q.base += total;
}

// The tree of block_sum over a 256-thread block's eight warp sums.
__device__ __forceinline__ double coop_block_tree(const double *p) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __ldcg(p + i);
    return ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
}

// block_sum<256> over the first 256 threads of a larger block; in thread 0.
__device__ __forceinline__ double coop_sum256(double v, double *sh) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && threadIdx.x < kBlock) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = threadIdx.x < kBlock / 32 ? sh[threadIdx.x] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

// Threads per block for n warps of items on `sms` blocks: enough for one pass, 256,
// 512 or 1,024 (us a substep with 256, 512 and 1,024: 5k particles in 2D, 16 warps of
// lanes a block, 105 / 83 / 85; 8k in 3D, 16 warps, 124 / 96 / 93; 1.3k, 8 warps and
// one for the boundary, 86 / 79 / 84).
inline int coop_threads(int64_t n_warps, int sms) {
    const int64_t per = (n_warps + sms - 1) / sms;
    return per <= 8 ? 256 : per <= 16 ? 512 : 1024;
}

// A cooperative launch of one block per SM.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_coop(void (*kernel)(KArgs...), int sms, int threads, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace tsph
