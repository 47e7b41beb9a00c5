// VFSPH volume-fraction update (the reference's "FBM" block), sph.py:301-379,
// driven as in main.py:244-250 (commented out there; enabled by fbm_enabled):
//
//   while general_flag:
//       clean_tmp; convect (drift velocities + convective flux); diffuse; check_tmp
//   update_volume_frac
//
// The drift velocities depend only on the step's velocities and volume
// fractions, which no pass changes, so they are computed once.  A pass sums the
// convective and diffusive flux of each unflagged particle over its unflagged
// neighbours and flags it if any phase would go negative; flags set during pass
// p (value p) do not exclude a neighbour until pass p + 1, which is what the
// reference's separate check kernel achieves.  Each scene runs its own pass
// loop; the graph loop runs while any scene does.  The number of passes is
// capped (fbm_max_passes); the reference loops forever if a flagged particle's
// own volume fraction is already negative.
#include <cuda_runtime.h>

#include "ctx.h"
#include "fbm.cuh"

namespace tsph {

__global__ void k_fbm_begin(KConst k, cudaGraphConditionalHandle h, int use_cond) {
    pdl_entry();
    __shared__ int any_sh;
    if (threadIdx.x == 0) any_sh = 0;
    __syncthreads();
    int any = 0;
    for (int s = threadIdx.x; s < k.n_scenes; s += blockDim.x) {
        SceneStep &st = k.ss[s];
        st.fbm_pass = 0;
        st.general_flag = 0;
        // SPH_clean_value sets general_flag = 1: at least one pass
        st.fbm_cond = k.sc[s].f_n > 0 ? 1 : 0;
        st.gflag_out = st.fbm_cond;
        any |= st.fbm_cond;
    }
    if (any) atomicOr(&any_sh, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        k.dg->fbm_any = any_sh;
        if (use_cond) cudaGraphSetConditional(h, any_sh ? 1u : 0u);
    }
}

template <int DIM, int P>
__global__ void __launch_bounds__(kBlock) k_fbm_drift(KConst k, FluidBuf F) {
    pdl_entry();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int sc = k.f_chunk_scene[(blockIdx.x * (int64_t)kBlock) / kChunk];
    const SceneConst &c = k.sc[sc];
    if (s - c.f_slot < c.f_n) fbm_drift_item<DIM, P>(k, F, sc, c, k.ss[sc].cur, s);
}

// One pass: SPH_FBM_clean_tmp + pair loop of SPH_FBM_convect + SPH_FBM_diffuse +
// SPH_FBM_check_tmp (sph.py:301-372).  The scene's last block evaluates its loop
// test; the grid's last block sets the graph condition.
// Up to two phases the pass is held to 48 registers (5 blocks per SM, measured
// faster); with more phases the per-phase arrays would spill.
template <int DIM, int P>
__global__ void __launch_bounds__(kBlock, P <= 2 ? 5 : 1) k_fbm_pass(KConst k, FluidBuf F, BoundBuf B,
                                                     cudaGraphConditionalHandle h, int use_cond) {
    pdl_entry();
    __shared__ int any_neg;
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int sc = k.f_chunk_scene[(blockIdx.x * (int64_t)kBlock) / kChunk];
    const SceneConst &c = k.sc[sc];
    SceneStep &st = k.ss[sc];
    const bool running = st.fbm_cond != 0;
    if (threadIdx.x == 0) any_neg = 0;
    __syncthreads();
    const int pass = st.fbm_pass + 1;
    if (running && s - c.f_slot < c.f_n) {
        if (fbm_pass_item<DIM, P, true, true>(k, F, B, sc, c, st, pass, s)) any_neg = 1;
    }
    __syncthreads();
    if (running) {
        if (threadIdx.x == 0 && any_neg) atomicExch(&st.general_flag, 1);
        const unsigned int nblk = (unsigned int)(c.f_slots / kBlock);
        if (last_block_done(&st.ticket[kStFbm], nblk)) {
            if (threadIdx.x == 0) {
                const int gf = atomicAdd(&st.general_flag, 0);
                st.fbm_pass = pass;
                st.fbm_passes = pass;
                st.gflag_out = gf;
                const int cond = gf && pass < c.fbm_max_passes;
                if (gf && !cond) st.status |= TSPH_ST_FBM_PASS_CAP;
                st.fbm_cond = cond;
                st.general_flag = 0;
                st.ticket[kStFbm] = 0;
            }
        }
    }
    if (last_block_done(&k.dg->ticket[kGtFbm], gridDim.x)) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int any = 0;
            for (int q = lane; q < k.n_scenes; q += 32) any |= (__ldcg(&k.ss[q].fbm_cond) != 0);
            any = __any_sync(0xffffffffu, any);
            if (lane == 0) {
                k.dg->fbm_any = any;
                k.dg->ticket[kGtFbm] = 0;
                if (use_cond) cudaGraphSetConditional(h, any ? 1u : 0u);
            }
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_fbm_redo(FluidBuf F, int pass) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < F.cap) F.redo[(pass & 1) * F.cap + s] = pass;
}

template <int P>
static void fbm_pass_dim(tsph_ctx &c, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st, bool drift) {
    const int nb = blocks_for(c.F.cap);
    if (c.k.dim == 3) {
        if (drift) TSPH_LAUNCH((k_fbm_drift<3, P>), nb, kBlock, st, c.k, c.F);
        else TSPH_LAUNCH((k_fbm_pass<3, P>), nb, kBlock, st, c.k, c.F, c.B, h, use_cond);
    } else {
        if (drift) TSPH_LAUNCH((k_fbm_drift<2, P>), nb, kBlock, st, c.k, c.F);
        else TSPH_LAUNCH((k_fbm_pass<2, P>), nb, kBlock, st, c.k, c.F, c.B, h, use_cond);
    }
}

static void fbm_dispatch(tsph_ctx &c, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st, bool drift) {
    switch (c.k.P) {
        case 1: fbm_pass_dim<1>(c, h, use_cond, st, drift); break;
        case 2: fbm_pass_dim<2>(c, h, use_cond, st, drift); break;
        case 3: fbm_pass_dim<3>(c, h, use_cond, st, drift); break;
        case 4: fbm_pass_dim<4>(c, h, use_cond, st, drift); break;
        case 5: fbm_pass_dim<5>(c, h, use_cond, st, drift); break;
        case 6: fbm_pass_dim<6>(c, h, use_cond, st, drift); break;
        case 7: fbm_pass_dim<7>(c, h, use_cond, st, drift); break;
        default: fbm_pass_dim<8>(c, h, use_cond, st, drift); break;
    }
}

void launch_fbm_begin(tsph_ctx &c, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st) {
    cudaMemsetAsync(c.F.flagpass, 0, sizeof(int) * c.F.cap, st);
    c.launches += 2;
    fbm_dispatch(c, 0, 0, st, true);
    TSPH_LAUNCH((k_fbm_begin), 1, 256, st, c.k, h, use_cond);
}

void launch_fbm_pass(tsph_ctx &c, cudaGraphConditionalHandle h, int use_cond, cudaStream_t st) {
    c.launches += 1;
    fbm_dispatch(c, h, use_cond, st, false);
}

void launch_fbm_redo(tsph_ctx &c, int pass, cudaStream_t st) {
    k_fbm_redo<<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.F, pass);
}

}  // namespace tsph
