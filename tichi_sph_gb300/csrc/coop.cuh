// Pieces of the cooperative kernels: the grid-wide barrier, each block's share of the
// items, sums in the order of the separate kernels, the launch.
#pragma once

#include <utility>

#include "ctx.h"

namespace tsph {

// A poll of the barrier's counter takes about half a microsecond: the limit is
// a few seconds, after which the step is given up and its status says so.
constexpr unsigned int kSpinLimit = 1u << 23;

// Barrier over the grid's blocks (all resident: a cooperative launch).  The
// counter only grows within a launch; the launch's last block to leave sets it
// back.  False: a block did not arrive within the limit; every block then leaves.
struct GridBarrier {
    unsigned int *bar;  // words kBarCount, kBarGaveUp, kBarLeft
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
                if (n > kSpinLimit) atomicExch(bar + kBarGaveUp, 1u);
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
    int64_t first, last;  // runs [first, last)
    __device__ __forceinline__ WarpShare(int64_t n) {
        const unsigned int nw = (unsigned int)((n + 31) >> 5), per = nw / gridDim.x, more = nw % gridDim.x;
        first = (int64_t)blockIdx.x * per + min(blockIdx.x, more);
        last = first + per + (blockIdx.x < more ? 1 : 0);
    }
    __device__ __forceinline__ int64_t count() const { return last - first; }
};

// Runs ff(i, warp) over the fluid's nf items and fb(i) over the boundary's nb in
// the block's warps (every lane of a warp calls, i may be past the end).
template <class FF, class FB>
__device__ __forceinline__ void for_items(int64_t nf, int64_t nb, FF &&ff, FB &&fb) {
    const WarpShare f(nf), b(nb);
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int64_t total = f.count() + b.count();
    for (int64_t w = threadIdx.x >> 5; w < total; w += warps) {
        if (w < f.count()) ff((f.first + w) * 32 + lane, f.first + w);
        else fb((b.first + w - f.count()) * 32 + lane);
    }
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
// 512 or 1,024 (fewer warps meet sooner at a barrier: a substep of 5k particles
// takes 136 us with 8 warps a block, 145 with 32).
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
