// Recording hooks of the forward step: kernels of their own in adjoint.cu, inside
// the one-launch step of small scenes (small.cu).
#pragma once

#include "ctx.h"
#include "tape.h"

namespace tsph {

// Recording hooks of the forward step, per particle; `slot` is the tape slot.
// The state after the density sweep, fluid slot s (slot 0 records the scalars).
__device__ __forceinline__ void tape_state_fluid_item(const KConst &k, const FluidBuf &F, const TapeArrays &a,
                                                      int slot, int64_t s) {
    const SceneConst &c = k.s0;
    const SceneStep &st = k.ss[0];
    TapeMeta &m = a.meta[slot];
    if (s < c.f_n) {
        const int64_t o = slot * a.cap + s;
        a.perm[o] = F.perm[s];
        a.pos[o] = F.pos[s];
        a.mpsi[o] = F.mpsi[s];
        a.a1[o] = F.a1[s];
        a.a2[o] = F.dens[s].w;
        a.rho0[o] = F.rho0[s];
        if (a.vf0) a.vf0[o] = F.vf[s];
        const unsigned int pc = F.nbr_cnt[s];
        a.cnt[o] = pc;
        if (pc == kNbrOverflow) {
            atomicOr(&m.status, TSPH_TAPE_LIST_OVERFLOW);
        } else {
            const int nb4 = ((int)(pc & 0xffffu) + (int)(pc >> 16) + 3) >> 2;
            const int4 *src = reinterpret_cast<const int4 *>(F.nbr) + s;
            int4 *dst = reinterpret_cast<int4 *>(a.nbr + (int64_t)slot * a.nbr_max * a.cap) + s;
            for (int b = 0; b < nb4; ++b) dst[(int64_t)b * a.cap] = src[(int64_t)b * F.cap];
        }
    }
    if (s == 0) {
        m.n = (int32_t)c.f_n;
        m.nb = (int32_t)c.b_n;
        m.f_in = st.f_in;
        m.dt = k.sp[0].dt;
        m.mu = c.mu;
        if (st.f_in != c.f_n) atomicOr(&m.status, TSPH_TAPE_OUTSIDE_GRID);
    }
}

__device__ __forceinline__ void tape_state_bound_item(const KConst &k, const BoundBuf &B, const TapeArrays &a,
                                                      int slot, int64_t s) {
    if (s >= k.s0.b_n) return;
    const int64_t o = slot * a.bcap + s;
    a.bpos[o] = B.pos[s];
    a.bvel[o] = B.vadv[s];
    if (B.kappa[s] != 0.f) atomicOr(&a.meta[slot].status, TSPH_TAPE_BOUND_PSI);
}

// The iterate u^k read by the psi sweep and the kappa it wrote (between the two
// sweeps of iteration `it`).
__device__ __forceinline__ void tape_iter_item(const KConst &k, const FluidBuf &F, const TapeArrays &a, int slot,
                                               int kind, int it, int cur, int64_t s) {
    if (it >= a.max_iters) {
        if (s == 0) atomicOr(&a.meta[slot].status, TSPH_TAPE_ITER_OVERFLOW);
        return;
    }
    if (s >= k.s0.f_n) return;
    const int64_t o = (((int64_t)slot * 2 + kind) * a.max_iters + it) * a.cap + s;
    a.u[o] = F.vadv[cur * F.cap + s];
    a.kap[o] = F.kappa[s];
}

__device__ __forceinline__ void tape_vmid_item(const KConst &k, const FluidBuf &F, const TapeArrays &a, int slot,
                                               int64_t s) {
    if (s >= k.s0.f_n) return;
    a.vmid[slot * a.cap + s] = F.vel[s];
    if (a.nrm) a.nrm[slot * a.cap + s] = F.normal[s];
}

__device__ __forceinline__ void tape_end_item(const KConst &k, const TapeArrays &a, int slot) {
    TapeMeta &m = a.meta[slot];
    m.kd = k.ss[0].div_iter;
    m.kp = k.ss[0].incom_iter;
}

}  // namespace tsph
