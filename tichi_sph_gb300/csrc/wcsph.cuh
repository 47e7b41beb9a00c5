// Weakly compressible pressure block, per particle (wcsph.cu describes it): kernels
// of its own there, inside the one-launch step of small scenes (small.cu).
#pragma once

#include "ctx.h"

namespace tsph {

// (rho / rho0)^7 by squaring, as an integer power.
__device__ __forceinline__ float wc_pow7(float r) {
    const float r2 = r * r;
    const float r4 = r2 * r2;
    return r4 * r2 * r;
}

__device__ __forceinline__ void wc_pressure_fluid_item(const FluidBuf &F, const SceneConst &c, int64_t s) {
    const float rho = F.dens[s].y, rho0 = F.rho0[s];
    float p = (rho0 * (float)(c.cs * c.cs)) / (float)c.wc_gamma * (wc_pow7(rho / rho0) - 1.f);
    if (p < 0.f) p = 0.f;
    F.wcp[s] = make_float2(p, p / (rho * rho));
}

__device__ __forceinline__ void wc_pressure_bound_item(const BoundBuf &B, const float *bpress, int64_t s) {
    const float p = bpress ? bpress[B.perm[s]] : 0.f;
    const float rho = B.dens[s].y;
    B.wcp2[s] = p / (rho * rho);
}

template <int DIM, bool M, bool NC>
__device__ __forceinline__ void wc_acce_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                             const SceneConst &c, const SceneStep &st, int cur, int64_t s) {
    const float h2 = c.h2, inv_h = c.inv_h, sig_h = c.sig_h;
    const float4 pi = F.pos[s];
    const float pri = F.wcp[s].y;
    float ax = 0.f, ay = 0.f, az = 0.f;
    auto term = [&](float4 pj, float prj, float mj) {
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < h2 && r2 > 0.f) {
            float r;
            const float ri = pair_rinv(r2, r);  // rsqrt pair geometry, as the other sweeps
            const float f = -(pri + prj) * mj * (kwg(r * inv_h) * sig_h) * ri;
            ax += f * dx;
            ay += f * dy;
            az += f * dz;
        }
    };
    for_each_neighbor_tpp<DIM, true, 1, M, NC>(c, st, k.R, F, B, s, 0, pi,
        [&](int j, auto) { term(F.pos[j], F.wcp[j].y, F.mv[j].x); },
        [&](int j, auto) { term(B.pos[j], B.wcp2[j], B.mv[j].x); });
    const float4 a0 = F.acc[s];
    const float4 a = make_float4(a0.x + ax, a0.y + ay, a0.z + az, 0.f);
    F.acc[s] = a;
    const float dt = k.sp[sc].dt;
    const float4 v = F.vel[s];
    F.vadv[cur * F.cap + s] = make_float4(v.x + a.x * dt, v.y + a.y * dt, v.z + a.z * dt, 0.f);
}

}  // namespace tsph
