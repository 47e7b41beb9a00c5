// Neighbour sweeps of one substep as separate kernels: density + alpha, the Jacobi
// pair of the two pressure solves, and the advection forces (viscosity, surface
// tension).  What a particle does in each is in sweeps.cuh.
//
// One thread (or TPP threads) per particle in cell-sorted order; a block never
// straddles two scenes, so every block reads one scene's constants.  The
// density sweep scans the (2r+1)^dim template rows of the fluid grid and, where
// the reference pairs with the boundary set, of the boundary grid
// (visit_hits_r1 for radius 1, else visit_candidates), and records every pair with 0 < r < h in the fluid
// particle's neighbour list.  The later sweeps of the step walk that list
// (for_each_neighbor_tpp) -- about 30 entries instead of about 220 candidates in
// 3D -- in the same order.  Per-particle sums are FP32 (the reference's
// precision); global sums are FP64 with a fixed summation order.
//
// Solver loops run per scene: a scene's loop state (iteration, condition,
// v_adv buffer) lives in its SceneStep; blocks of a scene whose loop has ended
// do nothing, the last block of a scene evaluates its loop test, and the last
// block of the grid sets the CUDA-graph while condition to "any scene running".
#include <cuda_runtime.h>

#include "ctx.h"
#include "sweeps.cuh"

namespace tsph {

// True for the warp of this block that finishes last (every warp must call it).
__device__ __forceinline__ bool block_last_warp(unsigned int *arrived) {
    unsigned int old = 0;
    if ((threadIdx.x & 31) == 0) {
        __threadfence_block();
        old = atomicAdd(arrived, 1u);
    }
    old = __shfl_sync(0xffffffffu, old, 0);
    const bool last = old == blockDim.x / 32 - 1;
    if (last) __threadfence_block();
    return last;
}

// The last warp of the grid: OR of the scenes' loop conditions into cond_any and
// the graph condition.
__device__ __forceinline__ void publish_any(const KConst &k, int SceneStep::*field, int32_t *any_out,
                                            cudaGraphConditionalHandle h, int use_cond) {
    const int lane = threadIdx.x & 31;
    int any = 0;
    for (int s = lane; s < k.n_scenes; s += 32) any |= (__ldcg(&(k.ss[s].*field)) != 0);
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) {
        *any_out = any;
        if (use_cond) cudaGraphSetConditional(h, any ? 1u : 0u);
    }
}

// ----------------------------------------------------------------------------- density
template <int DIM, bool M, bool R1>
__global__ void __launch_bounds__(kBlock, 4) k_density_fluid(const __grid_constant__ KConst k,
                                                             const __grid_constant__ FluidBuf F,
                                                             const __grid_constant__ BoundBuf B, double *partials) {
    pdl_entry();
    __shared__ double sh[kBlock / 32];
    __shared__ unsigned int arrived;
    if (threadIdx.x == 0) arrived = 0;
    __syncthreads();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int sc = f_block_scene<M>(k, blockIdx.x * (int64_t)kBlock);
    const SceneConst &c = scene<M>(k, sc);
    SceneStep &st = k.ss[sc];
    const bool psi0 = density_does_psi(c, k.sp[sc].compression);
    double contrib = 0.0;
    if (s - c.f_slot < c.f_n)
        contrib = density_fluid_item<DIM, M, R1, true>(k, F, B, sc, c, st, st.cur, psi0, s);
    if (!psi0) return;  // uniform over the block (one scene)
    double bsum;
    if (block_sum_last_warp<kBlock>(contrib, sh, &arrived, bsum)) {
        if ((threadIdx.x & 31) == 0) partials[blockIdx.x] = bsum;
        const int64_t b0 = c.f_slot / kBlock;
        const unsigned int nblk = (unsigned int)(c.f_slots / kBlock);
        if (last_warp_done(&st.ticket[kStPsi], nblk)) {
            const int lane = threadIdx.x & 31;
            double v = 0.0;
            for (int64_t i = lane; i < (int64_t)nblk; i += 32) v += __ldcg(partials + b0 + i);
            v = warp_sum(v);
            if (lane == 0) {
                st.psi_sum = v;
                st.ticket[kStPsi] = 0;
                st.psi_ready = 1;
            }
        }
    }
}

template <int DIM, bool M, bool R1>
__global__ void __launch_bounds__(kBlock, 6) k_density_bound(KConst k, FluidBuf F, BoundBuf B) {
    pdl_entry();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int sc = b_block_scene<M>(k, blockIdx.x * (int64_t)kBlock);
    const SceneConst &c = scene<M>(k, sc);
    if (s - c.b_slot >= c.b_n) return;
    density_bound_item<DIM, M, R1, true>(k, F, B, c, k.ss[sc], k.sp[sc], s);
}

// ----------------------------------------------------------------------------- solver
// Sets every scene's loop condition before a solve: main.py:201 / main.py:222
// test `iter < iter_min or compression > tol` with the compression left by the
// previous solve.  A scene without fluid runs min(iter_min, iter_max + 1) empty
// iterations in the reference and its compression becomes 0/0 = NaN
// (sph.py:226); that is settled here without device work.  `flip` makes the
// v_adv written by the advection sweep current.
__global__ void k_solve_begin(KConst k, int kind, int flip, cudaGraphConditionalHandle h, int use_cond) {
    pdl_entry();
    __shared__ int any_sh;
    if (threadIdx.x == 0) any_sh = 0;
    __syncthreads();
    int any = 0;
    for (int s = threadIdx.x; s < k.n_scenes; s += blockDim.x) {
        const SceneConst &c = k.sc[s];
        SceneStep &st = k.ss[s];
        ScenePersist &sp = k.sp[s];
        const double tol = kind == kSolveDiv ? (double)c.div_tol : (double)c.comp_tol;
        int cond, it = 0;
        if (c.f_n > 0) {
            cond = (0 < c.iter_min) || (sp.compression > tol);
        } else {
            cond = 0;
            while (it < c.iter_min) {
                ++it;
                if (it > c.iter_max) break;
            }
            if (it > 0) sp.compression = __longlong_as_double(0x7ff8000000000000ll);
        }
        st.iter = it;
        st.cond = cond;
        if (kind == kSolveDiv) st.div_iter = it;
        else st.incom_iter = it;
        // the density sweep's first-iteration psi belongs to the divergence solve
        if (kind == kSolveDens) st.psi_ready = 0;
        if (flip) st.cur = 1 - st.cur;
        any |= cond;
    }
    if (any) atomicOr(&any_sh, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        k.dg->cond_any = any_sh;
        if (use_cond) cudaGraphSetConditional(h, any_sh ? 1u : 0u);
    }
}

// Sweep A: IPPE_adv_psi_init + IPPE_adv_psi (f,f)(f,b) + IPPE_psi_adv_non_negative
// (sph.py:196-226), TPP threads per particle.  Writes psi_adv and kappa =
// psi_adv / alpha; the scene's sum of psi_adv / psi0 goes to per-block partials
// and, through the scene's last block, to its psi_sum (block order:
// deterministic).  force = 1: the host runs the loop (kernel-level calls), so
// the sweep runs whatever the device-side loop condition says.
template <int DIM, int TPP, bool M>
__global__ void __launch_bounds__(kBlock, 6) k_psi(KConst k, FluidBuf F, BoundBuf B, double *partials, int force) {
    pdl_entry();
    __shared__ double sh[kBlock / 32];
    __shared__ unsigned int arrived;
    const int64_t first = blockIdx.x * (int64_t)(kBlock / TPP);
    const int sc = f_block_scene<M>(k, first);
    SceneStep &st = k.ss[sc];
    if (!st.cond && !force) return;  // this scene's loop has ended (uniform over the block)
    if (st.psi_ready) return;  // this iteration's sweep ran inside the density sweep
    if (threadIdx.x == 0) arrived = 0;
    __syncthreads();
    const SceneConst &c = scene<M>(k, sc);
    const Lanes<TPP> ln;
    const double contrib =
        psi_item<DIM, TPP, M, true>(k, F, B, sc, c, st, st.cur, ln, ln.s, ln.s - c.f_slot < c.f_n);
    double bsum;
    if (block_sum_last_warp<kBlock>(contrib, sh, &arrived, bsum)) {
        if ((threadIdx.x & 31) == 0) partials[blockIdx.x] = bsum;
        const int64_t b0 = c.f_slot * TPP / kBlock;
        const unsigned int nblk = (unsigned int)(c.f_slots * TPP / kBlock);
        if (last_warp_done(&st.ticket[kStPsi], nblk)) {
            const int lane = threadIdx.x & 31;
            double v = 0.0;
            for (int64_t i = lane; i < (int64_t)nblk; i += 32) v += __ldcg(partials + b0 + i);
            v = warp_sum(v);
            if (lane == 0) {
                st.psi_sum = v;
                st.ticket[kStPsi] = 0;
            }
        }
    }
}

// Sweep B: IPPE_update_vel_adv (f,f)(f,b), sph.py:229-244, into the scene's other
// v_adv buffer, TPP threads per particle.  The scene's last block evaluates the
// loop test of main.py:201-213 / 222-234 from sweep A's sum; the grid's last
// block sets the graph's while-node condition.  force = 1 (kernel-level calls,
// the host runs the loop): the sweep runs regardless of the device-side
// condition and leaves the loop test and its cap to the host.
template <int DIM, int TPP, bool M>
__global__ void __launch_bounds__(kBlock) k_vel(KConst k, FluidBuf F, BoundBuf B, int kind,
                                                cudaGraphConditionalHandle h, int use_cond, int force) {
    pdl_entry();
    __shared__ unsigned int arrived;
    if (threadIdx.x == 0) arrived = 0;
    __syncthreads();
    const int64_t first = blockIdx.x * (int64_t)(kBlock / TPP);
    const int sc = f_block_scene<M>(k, first);
    SceneStep &st = k.ss[sc];
    const SceneConst &c = scene<M>(k, sc);
    const bool running = force || st.cond != 0;
    if (running) {
        const Lanes<TPP> ln;
        vel_item<DIM, TPP, M, true>(k, F, B, sc, c, st, st.cur, ln, ln.s, ln.s - c.f_slot < c.f_n);
    }
    if (!block_last_warp(&arrived)) return;
    if (running) {
        const unsigned int nblk = (unsigned int)(c.f_slots * TPP / kBlock);
        if (last_warp_done(&st.ticket[kStVel], nblk) && (threadIdx.x & 31) == 0) {
            ScenePersist &sp = k.sp[sc];
            const double comp = st.psi_sum / (double)c.f_n;
            sp.compression = comp;
            const int it = st.iter + 1;
            st.iter = it;
            if (kind == kSolveDiv) st.div_iter = it;
            else st.incom_iter = it;
            if (!force) {
                const double tol = kind == kSolveDiv ? (double)c.div_tol : (double)c.comp_tol;
                const int capped = it > c.iter_max;
                const int cond = !capped && (it < c.iter_min || comp > tol);
                if (capped) st.status |= (kind == kSolveDiv ? TSPH_ST_DIV_ITER_CAP : TSPH_ST_DENS_ITER_CAP);
                st.cond = cond;
            }
            st.cur = 1 - st.cur;
            st.psi_ready = 0;
            st.ticket[kStVel] = 0;
        }
    }
    if (last_warp_done(&k.dg->ticket[kGtVel], gridDim.x)) {
        publish_any(k, &SceneStep::cond, &k.dg->cond_any, h, use_cond);
        if ((threadIdx.x & 31) == 0) k.dg->ticket[kGtVel] = 0;
    }
}

// ----------------------------------------------------------------------------- advection
template <int DIM, int TPP, bool M>
__global__ void __launch_bounds__(kBlock) k_normal(KConst k, FluidBuf F, BoundBuf B) {
    pdl_entry();
    const int64_t first = blockIdx.x * (int64_t)(kBlock / TPP);
    const int sc = f_block_scene<M>(k, first);
    const SceneConst &c = scene<M>(k, sc);
    const SceneStep &st = k.ss[sc];
    const Lanes<TPP> ln;
    normal_item<DIM, TPP, M, true>(k, F, B, c, st, ln, ln.s, ln.s - c.f_slot < c.f_n);
}

// Held to 48 registers, 5 blocks per SM (64 batched scenes: 1,713 us a substep, 1,739
// with the 70 registers the batched instance takes unbounded).  Batched instances
// with surface tension spill up to 236 bytes so and are faster all the same (the
// phase, unbounded before and now, us, with one and eight lanes: 16 scenes of 64k
// 583 / 412 and 1301 / 823, 32 of 4.9k in 2D 37 / 28 and 104 / 72).
template <int DIM, bool ST, int TPP, bool M>
__global__ void __launch_bounds__(kBlock, 5) k_advect(KConst k, FluidBuf F, BoundBuf B, float gs, float vs) {
    pdl_entry();
    const int64_t first = blockIdx.x * (int64_t)(kBlock / TPP);
    const int sc = f_block_scene<M>(k, first);
    const SceneConst &c = scene<M>(k, sc);
    const SceneStep &st = k.ss[sc];
    const Lanes<TPP> ln;
    advect_item<DIM, ST, TPP, M, true>(k, F, B, sc, c, st, st.cur, ln, ln.s, ln.s - c.f_slot < c.f_n, gs, vs);
}

// ----------------------------------------------------------------------------- launchers
// One-scene (M = false) or batched (M = true) kernel instances.
#define TSPH_M_DISPATCH(MULTI, ...)                                       \
    if (MULTI) { constexpr bool M = true; __VA_ARGS__; }                   \
    else { constexpr bool M = false; __VA_ARGS__; }

template <bool M, bool R1>
static void launch_density_r1(tsph_ctx &c, cudaStream_t st, cudaStream_t sd) {
    if (c.k.dim == 3) {
        TSPH_LAUNCH((k_density_bound<3, M, R1>), blocks_for(c.B.cap), kBlock, sd, c.k, c.F, c.B);
        TSPH_LAUNCH((k_density_fluid<3, M, R1>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B, c.S.partials);
    } else {
        TSPH_LAUNCH((k_density_bound<2, M, R1>), blocks_for(c.B.cap), kBlock, sd, c.k, c.F, c.B);
        TSPH_LAUNCH((k_density_fluid<2, M, R1>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B, c.S.partials);
    }
}

// The boundary particles' own sums run on the side stream beside the fluid
// sweep: neither writes what the other reads.
void launch_density(tsph_ctx &c, cudaStream_t st) {
    c.launches += 2;
    cudaStream_t sd = c.side ? c.side : st;
    fork_side(c, st);
    TSPH_M_DISPATCH(c.n_scenes > 1,
        if (c.scan_r1) launch_density_r1<M, true>(c, st, sd);
        else launch_density_r1<M, false>(c, st, sd);)
    join_side(c, st);
}

// Measurement only: lets the next psi sweep run in full although the density
// sweep did its first iteration's work.
__global__ void k_clear_psi_ready(KConst k) {
    pdl_entry();
    for (int s = threadIdx.x; s < k.n_scenes; s += blockDim.x) k.ss[s].psi_ready = 0;
}

void launch_clear_psi_ready(tsph_ctx &c, cudaStream_t st) { TSPH_LAUNCH((k_clear_psi_ready), 1, 256, st, c.k); }

__global__ void k_status_or(KConst k, int bits) {
    pdl_entry();
    atomicOr(&k.ss[0].status, bits);
}

void launch_status_or(tsph_ctx &c, int bits, cudaStream_t st) { TSPH_LAUNCH((k_status_or), 1, 1, st, c.k, bits); }

void launch_solve_begin(tsph_ctx &c, int kind, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st) {
    c.launches += 1;
    TSPH_LAUNCH((k_solve_begin), 1, 256, st, c.k, kind, kind == kSolveDens ? 1 : 0, h, use_cond);
}

// Threads per particle of the list sweeps (1, 2, 4 or 8); see Lanes.
#define TSPH_TPP_DISPATCH(TPP_VAL, ...)                                   \
    switch (TPP_VAL) {                                                     \
        case 2: { constexpr int TPP = 2; __VA_ARGS__; } break;             \
        case 4: { constexpr int TPP = 4; __VA_ARGS__; } break;             \
        case 8: { constexpr int TPP = 8; __VA_ARGS__; } break;             \
        default: { constexpr int TPP = 1; __VA_ARGS__; } break;            \
    }

static int tpp_blocks(int64_t slots, int tpp) { return blocks_for(slots * tpp); }

void launch_psi(tsph_ctx &c, cudaStream_t st, int force) {
    c.launches += 1;
    const int tpp = c.tpp;
    const int nb = tpp_blocks(c.F.cap, tpp);
    TSPH_M_DISPATCH(c.n_scenes > 1, TSPH_TPP_DISPATCH(tpp,
        if (c.k.dim == 3) TSPH_LAUNCH((k_psi<3, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, c.S.partials, force);
        else TSPH_LAUNCH((k_psi<2, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, c.S.partials, force)))
}

void launch_vel(tsph_ctx &c, int kind, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st, int force) {
    c.launches += 1;
    const int tpp = c.tpp;
    const int nb = tpp_blocks(c.F.cap, tpp);
    TSPH_M_DISPATCH(c.n_scenes > 1, TSPH_TPP_DISPATCH(tpp,
        if (c.k.dim == 3) TSPH_LAUNCH((k_vel<3, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, kind, h, use_cond, force);
        else TSPH_LAUNCH((k_vel<2, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, kind, h, use_cond, force)))
}

void launch_solve_iter(tsph_ctx &c, int kind, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st) {
    launch_psi(c, st);
    launch_vel(c, kind, h, use_cond, st);
}

void launch_advect(tsph_ctx &c, cudaStream_t st, int terms) {
    const int tpp = c.tpp;
    const int nb = tpp_blocks(c.F.cap, tpp);
    const bool st_on = c.st_on != 0 && (terms & TSPH_TERM_SURFACE_TENSION);
    const float gs = (terms & TSPH_TERM_GRAVITY) ? 1.f : 0.f, vs = (terms & TSPH_TERM_VISCOSITY) ? 1.f : 0.f;
    c.launches += st_on ? 2 : 1;
    TSPH_M_DISPATCH(c.n_scenes > 1, TSPH_TPP_DISPATCH(tpp,
        if (c.k.dim == 3) {
            if (st_on) {
                TSPH_LAUNCH((k_normal<3, TPP, M>), nb, kBlock, st, c.k, c.F, c.B);
                TSPH_LAUNCH((k_advect<3, true, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, gs, vs);
            } else {
                TSPH_LAUNCH((k_advect<3, false, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, gs, vs);
            }
        } else {
            if (st_on) {
                TSPH_LAUNCH((k_normal<2, TPP, M>), nb, kBlock, st, c.k, c.F, c.B);
                TSPH_LAUNCH((k_advect<2, true, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, gs, vs);
            } else {
                TSPH_LAUNCH((k_advect<2, false, TPP, M>), nb, kBlock, st, c.k, c.F, c.B, gs, vs);
            }
        }))
}

}  // namespace tsph
