// Grid build, gather and write-back of one substep, per particle.  The kernels of
// grid.cu run one of them over all particles; the one-launch step of small
// scenes (small.cu) runs them one after another.
#pragma once

#include "ctx.h"

namespace tsph {

// ----------------------------------------------------------------------------- encode
// Ngrid.encode, sph_obj.py:300-306: structured cell, scene-local linear code,
// count in the scene's range of the global grid.  A particle without a valid
// code gets a rank in its scene's tail.
template <int DIM>
__device__ __forceinline__ void encode_item(const KConst &k, const tsph_set &U, int sc, int *count, int *slot, int *tail,
                                            int *status, int64_t i) {
    Geo g;
    g.load(k.sc[sc], k.R);
    float4 p = make_float4(U.pos[i * DIM], U.pos[i * DIM + 1], DIM == 3 ? U.pos[i * DIM + 2] : 0.f, 0.f);
    bool ok;
    long long code = cell_code<DIM>(p, g, ok);
    const float c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int d = 0; d < DIM; ++d)
        U.neighb_cell_structured_seq[i * DIM + d] = ok ? (int)floorf(__fdiv_rn(c[d] - g.lb[d], g.h)) : 0;
    U.neighb_cell_seq[i] = (int)code;
    int s;
    if (ok && code > 0 && code < g.node_num) {
        s = atomicAdd(count + g.cbase + code, 1);
    } else {
        s = -1 - atomicAdd(tail, 1);
        atomicOr(status, ok ? TSPH_ST_OUTSIDE_GRID : (TSPH_ST_NONFINITE_POS | TSPH_ST_OUTSIDE_GRID));
    }
    slot[i] = s;
}

// ----------------------------------------------------------------------------- scatter
__device__ __forceinline__ void scatter_item(const KConst &k, int bound, const int *code, const int *slot,
                                             const int *start, int *perm, int64_t i) {
    const int sc = bound ? k.b_user_scene[i] : k.f_user_scene[i];
    const SceneConst &c = k.sc[sc];
    const SceneStep &st = k.ss[sc];
    const int sl = slot[i];
    long long s;
    if (sl >= 0) s = (long long)start[c.cbase + code[i]] + (bound ? st.b_shift : st.f_shift) + sl;
    else s = (bound ? c.b_slot + st.b_in : c.f_slot + st.f_in) + (-1 - sl);
    perm[s] = (int)i;
}

// Sorted slot of the particle `pid` found at unsorted slot range [beg, end) of
// its cell (or of its scene's tail of particles without a valid cell): a cell's
// particles are ordered by id, so its slot is the range's first slot plus the
// number of the range's particles with a smaller id.
__device__ __forceinline__ int64_t sorted_slot(const int *perm_u, int64_t beg, int64_t end, int pid) {
    int r = 0;
    for (int64_t a = beg; a < end; ++a) r += perm_u[a] < pid;
    return beg + r;
}

// The slot range of the cell (in-grid particles, slots [slot0, slot0 + n_in))
// or of the scene's tail that holds the particle at unsorted slot u; `shift`
// maps the grid's scan positions to the scene's slots, as in k_scatter.
__device__ __forceinline__ void slot_range(const SceneConst &c, long long shift, const int *start,
                                           int64_t u, int64_t slot0, int32_t n_in, int32_t n_tail, int code,
                                           int64_t &beg, int64_t &end) {
    if (u - slot0 < n_in) {
        beg = start[c.cbase + code] + shift;
        end = start[c.cbase + code + 1] + shift;
    } else {
        beg = slot0 + n_in;
        end = beg + n_tail;
    }
}

// ----------------------------------------------------------------------------- gather
// Copies the caller-order state into the sorted working arrays; v_adv = vel
// (SPH_vel_2_vel_adv, sph.py:253-256).  X / psi0 follow the solver aliases,
// sph_obj.py:65-73.
template <int DIM>
__device__ __forceinline__ void gather_fluid_item(const KConst &k, const tsph_set &U, const FluidBuf &F, const SceneConst &c,
                                                  const SceneStep &st, int64_t u) {
    const int pid = F.perm_u[u];
    int64_t beg, end;
    slot_range(c, st.f_shift, F.start, u, c.f_slot, st.f_in, st.f_tail, U.neighb_cell_seq[pid], beg, end);
    const int64_t s = sorted_slot(F.perm_u, beg, end, pid);
    F.perm[s] = pid;
    F.inv[pid] = (int)s;
    const float *p = U.pos + (int64_t)pid * DIM;
    const float *v = U.vel + (int64_t)pid * DIM;
    const float m = U.mass[pid], V = U.rest_volume[pid], r0 = U.rest_density[pid];
    F.pos[s] = make_float4(p[0], p[1], DIM == 3 ? p[2] : 0.f, k.vfsph ? V : m);
    F.mv[s] = make_float2(m, V);
    F.rho0[s] = r0;
    F.mpsi[s] = make_float4(m, 0.f, k.vfsph ? 1.f : r0, 0.f);
    F.vadv[s] = make_float4(v[0], v[1], DIM == 3 ? v[2] : 0.f, 0.f);
    for (int q = 0; q < k.P; ++q) F.vf[q * F.cap + s] = U.volume_frac[(int64_t)pid * k.P + q];
}

template <int DIM>
__device__ __forceinline__ void gather_bound_item(const KConst &k, const tsph_set &U, const BoundBuf &B, const SceneConst &c, int sc,
                                                  int64_t u) {
    const SceneStep &st = k.ss[sc];
    const int pid = B.perm_u[u];
    int64_t beg, end;
    slot_range(c, st.b_shift, B.start, u, c.b_slot, st.b_in, st.b_tail, U.neighb_cell_seq[pid], beg, end);
    const int64_t s = sorted_slot(B.perm_u, beg, end, pid);
    B.perm[s] = pid;
    B.inv[pid] = (int)s;
    const float *p = U.pos + (int64_t)pid * DIM;
    const float *va = U.vel_adv + (int64_t)pid * DIM;
    const float m = U.mass[pid], V = U.rest_volume[pid];
    const float4 np = make_float4(p[0], p[1], DIM == 3 ? p[2] : 0.f, k.vfsph ? V : m);
    const float4 op = B.pos[s];
    const float2 omv = B.mv[s];
    // the slot's previous contents: equal everywhere means the same sorted
    // order, grid and boundary-boundary sums as the previous gather.  A change
    // also drops the kept sums for good, so that a later step cannot take them
    // after a call that gathered without a density sweep (the neighbour stats)
    const bool same = __float_as_uint(op.x) == __float_as_uint(np.x) && __float_as_uint(op.y) == __float_as_uint(np.y) &&
                      __float_as_uint(op.z) == __float_as_uint(np.z) && __float_as_uint(op.w) == __float_as_uint(np.w) &&
                      __float_as_uint(omv.x) == __float_as_uint(m) && __float_as_uint(omv.y) == __float_as_uint(V);
    // one store per warp that saw a change (a warp lies in one scene's chunk),
    // none once the flag is up: every slot differs in a first gather or under
    // a moving boundary, and the stores would all go to one word
    const unsigned int changed = __ballot_sync(__activemask(), !same);
    if (changed && (threadIdx.x & 31) == __ffs(changed) - 1 && !__ldcg(&k.ss[sc].b_dirty)) {
        k.ss[sc].b_dirty = 1;
        k.sp[sc].bb_valid = 0;
    }
    B.pos[s] = np;
    B.mv[s] = make_float2(m, V);
    B.vadv[s] = make_float4(va[0], va[1], DIM == 3 ? va[2] : 0.f, 0.f);
    B.kappa[s] = U.psi_adv[pid];  // divided by alpha once alpha is known
}

// ----------------------------------------------------------------------------- update
// SPH_update_volume_frac, SPH_update_mass, SPH_update_pos and SPH_update_energy
// (sph.py:265-286, 375-379) in the caller's particle order: each thread gathers
// its particle's sorted state (inv) so that the ~20 per-particle result arrays
// are written coalesced.  Blocks walk each scene's caller range padded to whole
// blocks.  Energies: per-particle FP32 terms, FP64 block sums, the scene's
// blocks summed in order by the scene's last block.
template <int DIM>
__device__ __forceinline__ void update_fluid_item(const KConst &k, const tsph_set &U, const FluidBuf &F, int sc,
                                                  const SceneConst &c, const SceneStep &st, int cur,
                                                  const int *bstart, int fbm, int st_on, int64_t pid, double &ke,
                                                  double &pe) {
    const int64_t s = F.inv[pid];
    const float dt = k.sp[sc].dt;
    const float4 v = F.vadv[cur * F.cap + s];
    const float4 p = F.pos[s];
    const float4 dn = F.dens[s];
    const float V = F.mv[s].y;
    const int flagged = fbm ? (F.flagpass[s] != 0) : 0;
    float rho0 = 0.f;
    for (int q = 0; q < k.P; ++q) {
        float vf = F.vf[q * F.cap + s];
        if (fbm) {
            const float t = F.vftmp[q * F.cap + s];
            if (!flagged) vf += t;
            U.volume_frac[pid * k.P + q] = vf;
            U.volume_frac_tmp[pid * k.P + q] = t;
        }
        rho0 += c.rho_phase[q] * vf;
    }
    const float m = rho0 * V;
    const float np[3] = {p.x + v.x * dt, p.y + v.y * dt, p.z + v.z * dt};
    const float vv[3] = {v.x, v.y, v.z};
    const float4 acc = F.acc[s];
    const float aa[3] = {acc.x, acc.y, acc.z};
    const float4 a1 = F.a1[s];
    const float a1v[3] = {a1.x, a1.y, a1.z};
    const int64_t b = pid * DIM;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        U.pos[b + d] = np[d];
        U.vel[b + d] = vv[d];
        U.vel_adv[b + d] = vv[d];
        U.acce_adv[b + d] = aa[d];
        U.alpha_1[b + d] = a1v[d];
    }
    if (st_on) {
        const float4 nr = F.normal[s];
        const float nrv[3] = {nr.x, nr.y, nr.z};
#pragma unroll
        for (int d = 0; d < DIM; ++d) U.normal[b + d] = nrv[d];
    }
    if (fbm) {
        const float4 fa = F.facc[s];
        const float fav[3] = {fa.x, fa.y, fa.z};
#pragma unroll
        for (int d = 0; d < DIM; ++d) U.acce[b + d] = fav[d];
        for (int q = 0; q < k.P; ++q) {
            const float4 dv = F.drift[s * k.P + q];
            const float dvv[3] = {dv.x, dv.y, dv.z};
#pragma unroll
            for (int d = 0; d < DIM; ++d) U.drift_vel[(pid * k.P + q) * DIM + d] = dvv[d];
        }
        U.fbm_zeta[pid] = F.zeta[s];
    }
    U.flag[pid] = flagged;
    U.mass[pid] = m;
    U.rest_density[pid] = rho0;
    U.W[pid] = dn.x;
    U.sph_density[pid] = dn.y;
    U.sph_compression[pid] = dn.z;
    U.psi_adv[pid] = F.psiadv[s];
    if (F.wcp && U.pressure) U.pressure[pid] = F.wcp[s].x;
    U.alpha[pid] = a1.w;  // alpha, stored beside alpha_1 by the density sweep
    U.alpha_2[pid] = dn.w;
    if (s - c.f_slot < st.f_in) {
        // slot in the reference's combined grid: cell offset over both sets, fluid first
        const int code = U.neighb_cell_seq[pid];
        U.neighb_in_cell_seq[pid] = (int)(s - st.f_shift) + bstart[c.cbase + code];
    }
    float v2 = 0.f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) v2 += vv[d] * vv[d];
    ke = (double)(0.5f * m * v2);
    pe = (double)(-m * c.g[1] * (np[1] - c.lb[1]));
}

// Adds the finished step to the scene's running totals.
__device__ __forceinline__ void step_totals(ScenePersist &sp, const SceneStep &st) {
    sp.total_div_iter += st.div_iter;
    sp.total_incom_iter += st.incom_iter;
    sp.total_fbm_passes += st.fbm_passes;
    sp.max_dens_compression = fmax(sp.max_dens_compression, sp.compression);
    sp.steps += 1;
}

template <int DIM>
__device__ __forceinline__ void update_bound_item(const KConst &k, const tsph_set &U, const BoundBuf &B,
                                                  const int *fstart, int64_t pid) {
    const int sc = k.b_user_scene[pid];
    const SceneConst &c = k.sc[sc];
    const SceneStep &st = k.ss[sc];
    if (pid == c.b_user) {
        // the density sweep of this step has run: BoundBuf::bb holds the
        // boundary-boundary sums of the boundary as gathered
        k.sp[sc].bb_valid = 1;
        k.sp[sc].bb_n = c.b_n;
    }
    const int64_t s = B.inv[pid];
    const float4 d = B.dens[s];
    U.W[pid] = d.x;
    U.sph_density[pid] = d.y;
    U.sph_compression[pid] = d.z;
    U.alpha_2[pid] = d.w;
    U.alpha[pid] = B.alpha[s];
    if (s - c.b_slot < st.b_in) {
        const int code = U.neighb_cell_seq[pid];
        U.neighb_in_cell_seq[pid] = (int)(s - st.b_shift) + fstart[c.cbase + code + 1];
    }
}

}  // namespace tsph
