// VFSPH volume-fraction update, per particle: the kernels of fbm.cu run one of these
// over all particles, the one-launch step of small scenes (small.cu) one after
// another.
#pragma once

#include "ctx.h"

namespace tsph {

// First loop of SPH_FBM_convect, sph.py:331-345.
template <int DIM, int P>
__device__ __forceinline__ void fbm_drift_item(const KConst &k, const FluidBuf &F, int sc, const SceneConst &c,
                                               int cur, int64_t s) {
    const float dt = k.sp[sc].dt;
    const float4 va = F.vadv[cur * F.cap + s];
    const float4 v = F.vel[s];
    const float ax = (va.x - v.x) / dt, ay = (va.y - v.y) / dt, az = (va.z - v.z) / dt;
    const float rho0 = F.rho0[s];
    float vf[P];
    float zeta = 0.f;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        vf[q] = F.vf[q * F.cap + s];
        zeta += vf[q] * (c.rho_phase[q] - rho0) / c.rho_phase[q];
    }
    const float gz = DIM == 3 ? c.g[2] : 0.f;
    const float fx = (ax - zeta * c.g[0]) / (1.f - zeta);
    const float fy = (ay - zeta * c.g[1]) / (1.f - zeta);
    const float fz = (az - zeta * gz) / (1.f - zeta);
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const float cq = vf[q] * (c.rho_phase[q] - rho0);
        float dx = cq * (c.g[0] - fx), dy = cq * (c.g[1] - fy), dz = cq * (gz - fz);
        const float w = vf[q] * c.rho_phase[q];
        if (w > 1e-6f) {
            dx /= w; dy /= w; dz /= w;
        } else {
            dx *= 0.f; dy *= 0.f; dz *= 0.f;
        }
        dx += fx - ax; dy += fy - ay; dz += fz - az;
        // w: the phase's volume fraction, which no pass changes (the passes
        // read a neighbour's drift and volume fraction in one load)
        F.drift[s * P + q] = make_float4(dx * dt, dy * dt, dz * dt, vf[q]);
    }
    F.redo[s] = F.redo[F.cap + s] = 0;
    F.acc[s] = make_float4(ax, ay, az, 0.f);
    F.facc[s] = make_float4(fx, fy, fz, 0.f);
    F.zeta[s] = zeta;
}

// One pass of one particle: SPH_FBM_clean_tmp + pair loop of SPH_FBM_convect +
// SPH_FBM_diffuse + SPH_FBM_check_tmp (sph.py:301-372).  Flags the particle, and
// returns true, if a phase would go negative.
//
// After the first pass only particles with a neighbour flagged in the pass before
// have another sum (the flagged leave it); the others keep theirs, and that they
// were not flagged.  A newly flagged particle therefore asks its neighbours to
// redo theirs (two words per slot, by the pass's parity: a pass reads one while
// it writes the other).  A particle outside the grid is nobody's neighbour and
// redoes every pass.  Bound by the gathers of a pair (position, two drifts and,
// after the first pass, the flag).  At 2M particles five passes took 350 us each and
// now take 400, 345, 204, 88 and 51.
template <int DIM, int P, bool M, bool NC>
__device__ __forceinline__ bool fbm_pass_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                              const SceneConst &c, const SceneStep &st, int pass, int64_t s) {
    const int fp = F.flagpass[s];
    if (fp == 0 && pass > 1 && F.redo[(pass & 1) * F.cap + s] != pass && s - c.f_slot < st.f_in) return false;
    float tmp[P];
    float vfi[P];
#pragma unroll
    for (int q = 0; q < P; ++q) {
        tmp[q] = 0.f;
        vfi[q] = F.vf[q * F.cap + s];
    }
    if (fp == 0) {
        Geo g;
        g.load(c, k.R);
        const float dt = k.sp[sc].dt;
        const float4 pi = F.pos[s];
        float4 ui[P];
#pragma unroll
        for (int q = 0; q < P; ++q) ui[q] = F.drift[s * P + q];
        const float cc = c.fbm_c * dt, cd = dt * c.fbm_D, eps = 0.01f * g.h2;
        for_each_neighbor_tpp<DIM, false, 1, M, NC>(c, st, k.R, F, B, s, 0, pi,
            [&](int j, auto) {
                const float4 pj = F.pos[j];
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (!(r2 < g.h2 && r2 > 0.f)) return;
                if (pass > 1) {
                    const int fj = F.flagpass[j];
                    if (fj != 0 && fj != pass) return;
                }
                // pair geometry from rsqrt and a fast quotient (as the other
                // sweeps; within a few ulp)
                float r;
                const float ri = pair_rinv(r2, r);
                const float wg = kwg(r * g.inv_h) * g.sig_h;
                const float Vj = k.vfsph ? pj.w : F.mv[j].y;  // VFSPH: X = rest volume
                const float gx = dx * ri * wg, gy = dy * ri * wg, gz = dz * ri * wg;
                const float dif = cd != 0.f ? __fdividef(cd * Vj * r * wg, r2 + eps) : 0.f;
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    const float4 uj = F.drift[(int64_t)j * P + q];
                    const float vfj = uj.w;
                    const float fx = vfi[q] * ui[q].x + vfj * uj.x;
                    const float fy = vfi[q] * ui[q].y + vfj * uj.y;
                    const float fz = vfi[q] * ui[q].z + vfj * uj.z;
                    tmp[q] -= cc * Vj * (fx * gx + fy * gy + fz * gz);
                    if (cd != 0.f) tmp[q] += (vfi[q] - vfj) * dif;
                }
            },
            [&](int, auto) {});
    }
    bool neg = false;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        F.vftmp[q * F.cap + s] = tmp[q];
        if (vfi[q] + tmp[q] < 0.f) neg = true;
    }
    if (neg && fp == 0) {
        F.flagpass[s] = pass;
        int *redo = F.redo + ((pass + 1) & 1) * F.cap;
        for_each_neighbor_tpp<DIM, false, 1, M, NC>(c, st, k.R, F, B, s, 0, F.pos[s],
                                                    [&](int j, auto) { redo[j] = pass + 1; }, [&](int, auto) {});
    }
    return neg;
}

}  // namespace tsph
