// Cell grid build (counting sort) and the gather / scatter between the caller's
// particle order and the cell-sorted working order, per scene.
//
// Reference: Ngrid.clear_node / encode / mem_shift / fill_node, sph_obj.py:295-323,
// and the per-step bookkeeping of sph.py:22-47, 265-286.  Differences by design:
// the cell offsets are an ordered exclusive scan instead of an atomic bump
// (mem_shift), and particles inside a cell are ordered by particle id, so the
// layout -- and every FP32 sum over it -- is deterministic.
#include <cuda_runtime.h>

#include "ctx.h"
#include "grid.cuh"

namespace tsph {

// ----------------------------------------------------------------------------- CFL
// cfl_condition, sph.py:41-47, per scene: dt = part_size / cs, lowered to
// part_size / |v| * cfl_factor for |v| > 1e-4.  part_size / v * cfl is monotone
// in v, so the minimum over particles is attained at max |v|.
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_cfl(KConst k, const float *__restrict__ vel, int64_t n) {
    pdl_entry();
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * kBlock;
    // each warp keeps its running maximum for the scene it last saw and issues
    // one atomic when the scene changes (and at the end): one atomic per warp
    // for a one-scene context instead of one per warp and iteration
    int wsc = -1;
    float wmax = 0.f;
    for (int64_t base = blockIdx.x * (int64_t)kBlock; base < n; base += stride) {
        const int64_t i = base + threadIdx.x;
        const bool act = i < n;
        float vn = 0.f;
        int sc = -1;
        if (act) {
            float s = 0.f;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float v = vel[i * DIM + d];
                s += v * v;
            }
            vn = sqrtf(s);
            if (!(vn > 1e-4f)) vn = 0.f;  // NaN norms fail the test, as in the reference
            sc = k.f_user_scene[i];
        }
        const int sc0 = __shfl_sync(0xffffffffu, sc, 0);
        if (sc0 < 0) continue;  // no particle left in this warp
        if (__all_sync(0xffffffffu, !act || sc == sc0)) {
            float m = vn;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (sc0 != wsc) {
                if (lane == 0 && wsc >= 0 && wmax > 0.f) atomicMax(&k.ss[wsc].vmax_bits, __float_as_uint(wmax));
                wsc = sc0;
                wmax = m;
            } else {
                wmax = fmaxf(wmax, m);
            }
        } else if (act && vn > 0.f) {
            atomicMax(&k.ss[sc].vmax_bits, __float_as_uint(vn));
        }
    }
    if (lane == 0 && wsc >= 0 && wmax > 0.f) atomicMax(&k.ss[wsc].vmax_bits, __float_as_uint(wmax));
    if (last_block_done(&k.dg->ticket[kGtCfl], gridDim.x)) {
        for (int s = threadIdx.x; s < k.n_scenes; s += kBlock) {
            const SceneConst &c = k.sc[s];
            float dt = __fdiv_rn(c.part_size, (float)c.cs);
            const float vm = __uint_as_float(atomicExch(&k.ss[s].vmax_bits, 0u));
            if (vm > 1e-4f) dt = fminf(dt, __fmul_rn(__fdiv_rn(c.part_size, vm), c.cfl));
            k.sp[s].dt = dt;
            k.sp[s].time_count += (double)dt;
        }
        if (threadIdx.x == 0) k.dg->ticket[kGtCfl] = 0;
    }
}

// ----------------------------------------------------------------------------- encode
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_encode(KConst k, tsph_set U, int bound, int *__restrict__ count,
                                                   int *__restrict__ slot) {
    pdl_entry();
    const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (i >= U.n) return;
    const int sc = bound ? k.b_user_scene[i] : k.f_user_scene[i];
    SceneStep &st = k.ss[sc];
    encode_item<DIM>(k, U, sc, count, slot, bound ? &st.b_tail : &st.f_tail, &st.status, i);
}

// ----------------------------------------------------------------------------- scan
// Exclusive scan of the cell counts in two launches (blockIdx.y selects the
// fluid (0) or boundary (1) grid; 4096 cells per block):
//   k_scan_reduce: each block's total; the grid's last block to finish scans
//     the totals in place (a ticket, no block waits for another);
//   k_scan_down: each block scans its cells again and adds its offset; the last
//     block over both grids derives the per-scene shifts from the finished
//     starts.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

struct ScanArgs {
    const int *count[2];
    int *start[2];
    int *blocks[2];
    int64_t n;
};

__device__ __forceinline__ int block_excl_scan(int v, int *sh, int &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = (lane < kScanThreads / 32) ? sh[lane] : 0;
        int u = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= o) u += y;
        }
        sh[lane] = u - t;           // exclusive prefix of warp totals
        if (lane == 31) sh[32] = u;  // block total
    }
    __syncthreads();
    total = sh[32];
    int r = sh[w] + x - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(ScanArgs a, int nblocks, unsigned int *tickets) {
    pdl_entry();
    __shared__ int sh[33];
    const int g = blockIdx.y;
    const int64_t base = blockIdx.x * (int64_t)kScanTile + threadIdx.x * kScanItems;
    int sum = 0;
#pragma unroll
    for (int t = 0; t < kScanItems; ++t)
        if (base + t < a.n) sum += a.count[g][base + t];
    int total;
    block_excl_scan(sum, sh, total);
    if (threadIdx.x == 0) a.blocks[g][blockIdx.x] = total;
    if (!last_block_done(&tickets[g], (unsigned int)nblocks)) return;
    // this grid's block totals -> exclusive offsets, in place; [nblocks] = total
    int carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += kScanTile) {
        int v[kScanItems];
        int s = 0;
        const int i0 = b0 + threadIdx.x * kScanItems;
#pragma unroll
        for (int t = 0; t < kScanItems; ++t) {
            v[t] = (i0 + t < nblocks) ? __ldcg(&a.blocks[g][i0 + t]) : 0;
            s += v[t];
        }
        int tot;
        int run = block_excl_scan(s, sh, tot) + carry;
#pragma unroll
        for (int t = 0; t < kScanItems; ++t) {
            if (i0 + t < nblocks) a.blocks[g][i0 + t] = run;
            run += v[t];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) {
        a.blocks[g][nblocks] = carry;
        tickets[g] = 0;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_down(ScanArgs a, int nblocks, KConst k, unsigned int *ticket) {
    pdl_entry();
    __shared__ int sh[33];
    const int g = blockIdx.y;
    const int64_t base = blockIdx.x * (int64_t)kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int sum = 0;
#pragma unroll
    for (int t = 0; t < kScanItems; ++t) {
        v[t] = (base + t < a.n) ? a.count[g][base + t] : 0;
        sum += v[t];
    }
    int total;
    int run = block_excl_scan(sum, sh, total) + a.blocks[g][blockIdx.x];
#pragma unroll
    for (int t = 0; t < kScanItems; ++t) {
        if (base + t < a.n) a.start[g][base + t] = run;
        run += v[t];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.start[g][a.n] = a.blocks[g][nblocks];
    if (!last_block_done(ticket, 2u * (unsigned int)nblocks)) return;
    // per scene: in-grid counts and the shift from global scan positions to the
    // scene's sorted slots
    for (int s = threadIdx.x; s < k.n_scenes; s += blockDim.x) {
        const SceneConst &c = k.sc[s];
        SceneStep &st = k.ss[s];
        const int f0 = __ldcg(&a.start[0][c.cbase]), f1 = __ldcg(&a.start[0][c.cbase + c.node_num]);
        const int b0 = __ldcg(&a.start[1][c.cbase]), b1 = __ldcg(&a.start[1][c.cbase + c.node_num]);
        st.f_in = f1 - f0;
        st.b_in = b1 - b0;
        st.f_shift = c.f_slot - f0;
        st.b_shift = c.b_slot - b0;
    }
    if (threadIdx.x == 0) *ticket = 0;
}

// ----------------------------------------------------------------------------- scatter
__global__ void __launch_bounds__(kBlock) k_scatter(KConst k, int bound, int64_t n, const int *__restrict__ code,
                                                    const int *__restrict__ slot, const int *__restrict__ start,
                                                    int *__restrict__ perm) {
    pdl_entry();
    const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (i < n) scatter_item(k, bound, code, slot, start, perm, i);
}

// ----------------------------------------------------------------------------- gather
// gather_fluid_item / gather_bound_item over all slots
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_gather_fluid(KConst k, tsph_set U, FluidBuf F) {
    pdl_entry();
    const int64_t u = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (u >= F.cap) return;
    const int sc = k.f_chunk_scene[u / kChunk];
    const SceneConst &c = k.sc[sc];
    if (u - c.f_slot < c.f_n) gather_fluid_item<DIM>(k, U, F, c, k.ss[sc], u);
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_gather_bound(KConst k, tsph_set U, BoundBuf B) {
    pdl_entry();
    const int64_t u = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (u >= B.cap) return;
    const int sc = k.b_chunk_scene[u / kChunk];
    const SceneConst &c = k.sc[sc];
    if (u - c.b_slot < c.b_n) gather_bound_item<DIM>(k, U, B, c, sc, u);
}

// ----------------------------------------------------------------------------- update
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_update_fluid(KConst k, tsph_set U, FluidBuf F,
                                                         const int *__restrict__ bstart, double *partials, int fbm,
                                                         int st_on) {
    pdl_entry();
    __shared__ double sh[kBlock / 32];
    const int sc = k.f_ublock_scene[blockIdx.x];
    const SceneConst &c = k.sc[sc];
    SceneStep &st = k.ss[sc];
    const int64_t local = (blockIdx.x - c.f_ublk0) * (int64_t)kBlock + threadIdx.x;
    double ke = 0.0, pe = 0.0;
    if (local < c.f_n) {
        update_fluid_item<DIM>(k, U, F, sc, c, st, st.cur, bstart, fbm, st_on, c.f_user + local, ke, pe);
    }
    const double bke = block_sum<kBlock>(ke, sh);
    const double bpe = block_sum<kBlock>(pe, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = bke;
        partials[2 * blockIdx.x + 1] = bpe;
    }
    const unsigned int nblk = (unsigned int)c.f_ublks;
    if (last_block_done(&st.ticket[kStUpdate], nblk)) {
        const int64_t b0 = c.f_ublk0;
        double a = 0.0, b = 0.0;
        for (int64_t i = threadIdx.x; i < (int64_t)nblk; i += kBlock) {
            a += __ldcg(partials + 2 * (b0 + i));
            b += __ldcg(partials + 2 * (b0 + i) + 1);
        }
        a = block_sum<kBlock>(a, sh);
        b = block_sum<kBlock>(b, sh);
        if (threadIdx.x == 0) {
            st.kinetic_energy = a;
            st.potential_energy = b;
            st.ticket[kStUpdate] = 0;
            step_totals(k.sp[sc], st);
        }
    }
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_update_bound(KConst k, tsph_set U, BoundBuf B,
                                                         const int *__restrict__ fstart) {
    pdl_entry();
    const int64_t pid = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (pid < U.n) update_bound_item<DIM>(k, U, B, fstart, pid);
}

// ----------------------------------------------------------------------------- neighbours
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// Per particle: its neighbours with 0 < r < h in each set (FP32 q < 1, as the
// reference tests) and their order-independent hash, or -- cand != 0 -- the
// number of candidates the density sweep's scan visits in each grid (no hash).
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_neighbor_stats(KConst k, int bound, FluidBuf F, BoundBuf B,
                                                           int32_t *counts, uint64_t *hash, int cand) {
    pdl_entry();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int64_t cap = bound ? B.cap : F.cap;
    if (s >= cap) return;
    const int sc = bound ? k.b_chunk_scene[s / kChunk] : k.f_chunk_scene[s / kChunk];
    const SceneConst &c = k.sc[sc];
    if (s - (bound ? c.b_slot : c.f_slot) >= (bound ? c.b_n : c.f_n)) return;
    const SceneStep &st = k.ss[sc];
    Geo g;
    g.load(c, k.R);
    const float4 pi = bound ? B.pos[s] : F.pos[s];
    bool ok;
    const long long code = cell_code<DIM>(pi, g, ok);
    int cf = 0, cb = 0;
    uint64_t hsum = 0;
    if (ok) {
        // the density sweep's visitor (it records the pairs every later sweep
        // walks): its skipped rows and cells must hold no pair with r < h
        visit_candidates_within<DIM>(F.start, g, pi, code, st.f_shift, 0, [&](int j) {
            const float4 pj = F.pos[j];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (cand) {
                ++cf;
            } else if (r2 > 0.f && sqrtf(r2) * g.inv_h < 1.f) {
                ++cf;
                hsum += mix64((uint64_t)(uint32_t)F.perm[j]);
            }
        });
        visit_candidates_within<DIM>(B.start, g, pi, code, st.b_shift, 0, [&](int j) {
            const float4 pj = B.pos[j];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (cand) {
                ++cb;
            } else if (r2 > 0.f && sqrtf(r2) * g.inv_h < 1.f) {
                ++cb;
                hsum += mix64((1ull << 32) | (uint64_t)(uint32_t)B.perm[j]);
            }
        });
    }
    const int pid = bound ? B.perm[s] : F.perm[s];
    counts[2 * pid] = cf;
    counts[2 * pid + 1] = cb;
    if (hash) hash[pid] = hsum;
}

// ----------------------------------------------------------------------------- launchers
void fork_side(tsph_ctx &c, cudaStream_t st) {
    if (!c.side) return;
    cudaEventRecord(c.ev_fork, st);
    cudaStreamWaitEvent(c.side, c.ev_fork, 0);
}

void join_side(tsph_ctx &c, cudaStream_t st) {
    if (!c.side) return;
    cudaEventRecord(c.ev_join, c.side);
    cudaStreamWaitEvent(st, c.ev_join, 0);
}

void launch_step_begin(tsph_ctx &c, cudaStream_t st) {
    c.scalars_on_host = 0;
    cudaMemsetAsync(c.k.ss, 0, sizeof(SceneStep) * c.k.n_scenes, st);
    cudaMemsetAsync(c.k.dg, 0, sizeof(DevGlobal), st);
}

void launch_cfl(tsph_ctx &c, const tsph_set &f, cudaStream_t st) {
    int nb = blocks_for(f.n);
    if (nb < 1) nb = 1;
    if (nb > 4 * 152) nb = 4 * 152;
    c.scalars_on_host = 0;
    c.launches += 1;
    if (c.k.dim == 3) TSPH_LAUNCH((k_cfl<3>), nb, kBlock, st, c.k, f.vel, f.n);
    else TSPH_LAUNCH((k_cfl<2>), nb, kBlock, st, c.k, f.vel, f.n);
}

void launch_grid_build(tsph_ctx &c, const tsph_set &f, const tsph_set &b, cudaStream_t st, bool with_cfl) {
    const int64_t nn = c.k.total_nodes;
    // the boundary set's encode, scatter and gather run on the side stream,
    // beside the fluid's; the scans cover both grids in one launch
    cudaStream_t sd = c.side ? c.side : st;
    c.counts_zero = 0;
    c.launches += (f.n > 0) + (b.n > 0) + 2 + (f.n > 0) + (b.n > 0) + 2;
    fork_side(c, st);
    if (with_cfl) launch_cfl(c, f, sd);  // nothing before the first solve reads dt
    cudaMemsetAsync(c.B.count, 0, sizeof(int) * nn, sd);
    if (b.n > 0) {
        if (c.k.dim == 3) TSPH_LAUNCH((k_encode<3>), blocks_for(b.n), kBlock, sd, c.k, b, 1, c.B.count, c.B.slot);
        else TSPH_LAUNCH((k_encode<2>), blocks_for(b.n), kBlock, sd, c.k, b, 1, c.B.count, c.B.slot);
    }
    cudaMemsetAsync(c.F.count, 0, sizeof(int) * nn, st);
    if (f.n > 0) {
        if (c.k.dim == 3) TSPH_LAUNCH((k_encode<3>), blocks_for(f.n), kBlock, st, c.k, f, 0, c.F.count, c.F.slot);
        else TSPH_LAUNCH((k_encode<2>), blocks_for(f.n), kBlock, st, c.k, f, 0, c.F.count, c.F.slot);
    }
    join_side(c, st);
    ScanArgs sa;
    sa.count[0] = c.F.count; sa.count[1] = c.B.count;
    sa.start[0] = c.F.start; sa.start[1] = c.B.start;
    sa.blocks[0] = c.S.scan_blocks; sa.blocks[1] = c.S.scan_blocks + c.S.scan_len / 2;
    sa.n = nn;
    const int nblk = (int)((nn + kScanTile - 1) / kScanTile);
    TSPH_LAUNCH((k_scan_reduce), dim3(nblk, 2), kScanThreads, st, sa, nblk, c.k.dg->ticket + kGtScanF);
    TSPH_LAUNCH((k_scan_down), dim3(nblk, 2), kScanThreads, st, sa, nblk, c.k, c.k.dg->ticket + kGtScanDone);
    fork_side(c, st);
    if (b.n > 0) TSPH_LAUNCH((k_scatter), blocks_for(b.n), kBlock, sd, c.k, 1, b.n, b.neighb_cell_seq, c.B.slot, c.B.start, c.B.perm_u);
    if (f.n > 0) TSPH_LAUNCH((k_scatter), blocks_for(f.n), kBlock, st, c.k, 0, f.n, f.neighb_cell_seq, c.F.slot, c.F.start, c.F.perm_u);
    // each set's gather orders its cells by particle id as it copies (a
    // particle's slot is its rank among its cell's ids)
    if (c.k.dim == 3) {
        TSPH_LAUNCH((k_gather_bound<3>), blocks_for(c.B.cap), kBlock, sd, c.k, b, c.B);
        TSPH_LAUNCH((k_gather_fluid<3>), blocks_for(c.F.cap), kBlock, st, c.k, f, c.F);
    } else {
        TSPH_LAUNCH((k_gather_bound<2>), blocks_for(c.B.cap), kBlock, sd, c.k, b, c.B);
        TSPH_LAUNCH((k_gather_fluid<2>), blocks_for(c.F.cap), kBlock, st, c.k, f, c.F);
    }
    join_side(c, st);
}

void launch_unsort(tsph_ctx &c, const tsph_set &f, const tsph_set &b, cudaStream_t st) {
    const int fbm = c.p.fbm_enabled ? 1 : 0;
    const int st_on = c.st_on;
    // boundary: over the caller's count (the kernel returns past it); one block at least
    const int nbb = b.n > 0 ? blocks_for(b.n) : 1;
    c.launches += 2;
    cudaStream_t sd = c.side ? c.side : st;
    fork_side(c, st);
    if (c.k.dim == 3) {
        TSPH_LAUNCH((k_update_bound<3>), nbb, kBlock, sd, c.k, b, c.B, c.F.start);
        TSPH_LAUNCH((k_update_fluid<3>), (int)c.k.f_ublocks, kBlock, st, c.k, f, c.F, c.B.start, c.S.partials, fbm, st_on);
    } else {
        TSPH_LAUNCH((k_update_bound<2>), nbb, kBlock, sd, c.k, b, c.B, c.F.start);
        TSPH_LAUNCH((k_update_fluid<2>), (int)c.k.f_ublocks, kBlock, st, c.k, f, c.F, c.B.start, c.S.partials, fbm, st_on);
    }
    join_side(c, st);
}

void launch_neighbor_stats(tsph_ctx &c, int32_t *fc, uint64_t *fh, int32_t *bc, uint64_t *bh, int cand,
                           cudaStream_t st) {
    if (c.k.dim == 3) {
        k_neighbor_stats<3><<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.k, 0, c.F, c.B, fc, fh, cand);
        k_neighbor_stats<3><<<blocks_for(c.B.cap), kBlock, 0, st>>>(c.k, 1, c.F, c.B, bc, bh, cand);
    } else {
        k_neighbor_stats<2><<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.k, 0, c.F, c.B, fc, fh, cand);
        k_neighbor_stats<2><<<blocks_for(c.B.cap), kBlock, 0, st>>>(c.k, 1, c.F, c.B, bc, bh, cand);
    }
}

}  // namespace tsph
