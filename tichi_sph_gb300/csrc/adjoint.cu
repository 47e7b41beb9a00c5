// Hand-written reverse mode of the DFSPH substep.
//
// Forward (recorded): density + alpha (sph.py:50-105), the divergence-free
// Jacobi solve (main.py:199-214), gravity + viscosity (sph.py:108-129), the
// constant-density Jacobi solve (main.py:221-234) and the position update
// (sph.py:265-269), with dt, iteration counts and neighbour pairs fixed.
//
// Reverse, one thread per fluid particle in the recorded sorted order, every
// sweep a gather over the recorded neighbour list (no atomics; deterministic):
//
//   one Jacobi iteration u' = u - (1/(dt m_i)) sum_j (k_i X_j + k_j X_i) g_ij r_ij,
//   k = max(s, 0) / alpha, s_i = psi_i - psi0_i + dt sum_j X_j g_ij r_ij.(u_i - u_j)
//   (g(r) = W'(r)/r, r_ij = x_i - x_j) reverses into two sweeps with the
//   transposed structure -- the velocity update's adjoint is a divergence of
//   beta = lam_u' / (dt m) and the divergence's adjoint is a pressure-force-
//   shaped sum of lam_s:
//     k_adj_kappa: lam_k_i = -sum_j X_j g r_ij.(beta_i - beta_j) (- boundary),
//                  lam_s = [s > 0] lam_k / alpha, lam_alpha -= lam_k k / alpha,
//                  lam_psi += lam_s, lam_x += d/dx of the update's pair terms;
//     k_adj_vel:   lam_u = lam_u' + dt sum_j (lam_s_i X_j + lam_s_j X_i) g r_ij,
//                  lam_x += d/dx of the divergence's pair terms;
//   k_adj_visc reverses a = g + mu V(x, v, psi) (and yields dL/dmu);
//   k_adj_st1 / k_adj_st2 reverse the surface tension (sph.py:132-166): its
//     cohesion and curvature over the template candidates, then the normals;
//   k_adj_density reverses the density and alpha sums.
// The position derivative of a pair term g(r) r_ij . w is g w + (g'(r)/r)(r_ij . w) r_ij
// with g'(r)/r = (W''(r) - g(r)) / r^2.  Each pair appears in both particles'
// lists (fluid-fluid), so the terms a pair contributes through the other
// particle's sums are gathered too; boundary particles are static.
//
// The same formulas are restated in FP64 PyTorch in the autodiff oracle and
// checked there against torch.autograd and central finite differences.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <new>

#include "ctx.h"
#include "coop.cuh"
#include "tape.cuh"

namespace tsph {

void set_last_error_text(const char *msg);

namespace {

// w''(q) of the cubic spline (the derivative of kwg).
__device__ __forceinline__ float kwgg(float q) {
    return q <= 0.5f ? 6.f * (6.f * q - 2.f) : (q < 1.f ? 12.f * (1.f - q) : 0.f);
}

// Derivative of the cohesion spline shape kcoh: 3 q^2 (1 - q)^2 (1 - 2 q),
// doubled below q = 1/2.
__device__ __forceinline__ float kcohd(float q) {
    const float b = 1.f - q;
    const float t = 3.f * q * q * b * b * (1.f - 2.f * q);
    return q <= 0.5f ? 2.f * t : (q < 1.f ? t : 0.f);
}

// ----------------------------------------------------------------------------- recording
__global__ void k_tape_begin(TapeArrays a, int slot) {
    *a.dslot = slot;
    TapeMeta z;
    memset(&z, 0, sizeof(z));
    a.meta[slot] = z;
}

__global__ void __launch_bounds__(kBlock) k_tape_state(KConst k, FluidBuf F, BoundBuf B, TapeArrays a) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    tape_state_fluid_item(k, F, a, *a.dslot, s);
    tape_state_bound_item(k, B, a, *a.dslot, s);
}

__global__ void __launch_bounds__(kBlock) k_tape_iter(KConst k, FluidBuf F, int kind, TapeArrays a) {
    const SceneStep &st = k.ss[0];
    if (st.cond) tape_iter_item(k, F, a, *a.dslot, kind, st.iter, st.cur, blockIdx.x * (int64_t)kBlock + threadIdx.x);
}

__global__ void __launch_bounds__(kBlock) k_tape_vmid(KConst k, FluidBuf F, TapeArrays a) {
    tape_vmid_item(k, F, a, *a.dslot, blockIdx.x * (int64_t)kBlock + threadIdx.x);
}

// The fluid grid's cell starts of the recorded substep (surface tension on: its
// reverse visits the same template candidates as the forward).
__global__ void __launch_bounds__(kBlock) k_tape_start(FluidBuf F, TapeArrays a) {
    const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (i < a.nstart) a.start[(int64_t)(*a.dslot) * a.nstart + i] = F.start[i];
}

__global__ void k_tape_end(KConst k, TapeArrays a) { tape_end_item(k, a, *a.dslot); }

__global__ void __launch_bounds__(kBlock) k_density_out(KConst k, FluidBuf F, float *out) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s >= k.s0.f_n) return;
    out[F.perm[s]] = F.dens[s].y;
}

// ----------------------------------------------------------------------------- reverse
// One recorded slot, offset to its arrays.
struct SlotView {
    const int *perm;
    const float4 *pos, *mpsi, *a1, *vmid, *bpos, *bvel;
    const float *a2, *rho0;
    const unsigned int *cnt;
    const int *nbr;
    const float4 *u;     // [2][max_iters][cap]
    const float *kap;
    const float4 *nrm;   // surface tension on: normals, phase-0 volume fractions, cell starts
    const float *vf0;
    const int *start;
    Geo geo;
    int64_t cap;
    int n, max_iters;
    float dt, mu, h, h2, inv_h, sig_h, eps, gamma, c_coh;
};

// Pair geometry of r_ij = pi - pj (0 < r < h): g = W'(r)/r, G2 = g'(r)/r, W2 = W''(r).
struct Pair {
    float x, y, z, r2, g, G2, W2;
    __device__ __forceinline__ Pair(const SlotView &v, float4 pi, float4 pj) {
        x = pi.x - pj.x;
        y = pi.y - pj.y;
        z = pi.z - pj.z;
        r2 = x * x + y * y + z * z;
        // r and 1 / r from rsqrt, as the forward sweeps (within a few ulp)
        float r;
        const float ri = pair_rinv(r2, r);
        const float q = r * v.inv_h;
        g = kwg(q) * v.sig_h * ri;
        W2 = kwgg(q) * v.sig_h * v.inv_h;
        G2 = (W2 - g) * (ri * ri);
    }
    __device__ __forceinline__ float dot(float ax, float ay, float az) const { return x * ax + y * ay + z * az; }
};

// The recorded pairs of the particle at slot s, or of none for s beyond the last;
// its TPP lanes (ln) share them, a block of four entries each in turn.
template <int TPP, class FF, class FB>
__device__ __forceinline__ void for_pairs(const SlotView &v, const Lanes<TPP> &ln, int64_t s, FF &&ff, FB &&fb) {
    const unsigned int pc = s < v.n ? v.cnt[s] : 0u;
    const int nfl = (int)(pc & 0xffffu), nbo = (int)(pc >> 16);
    walk_blocks<TPP>(v.nbr, s, v.cap, ln.q, nfl, nfl + nbo, ff, fb);
}

// Working arrays of the reverse pass, in the slot's sorted order.
struct Lam {
    float4 *u, *u2;   // adjoint of the velocity (two buffers: the viscosity sweep); w: rest density
    float4 *x;        // of the position
    float4 *beta;     // lam_u / (dt m); w: kappa of the iteration to reverse next
    float4 *us;       // the iterate u^k; w: lam_s
    float4 *a1;       // of alpha's two sums
    float4 *n;        // of the surface normals
    float *psi, *alpha;
};

// Kappa of iteration `it` of a solve (it >= 0).
__device__ __forceinline__ const float *kappa_of(const SlotView &v, int kind, int it) {
    return v.kap + ((int64_t)kind * v.max_iters + it) * v.cap;
}

// lam_u of a particle as the next kappa sweep gathers it, with its kappa (it < 0:
// no sweep follows).
__device__ __forceinline__ void put_beta(const SlotView &v, const Lam &l, int kind, int it, float m, float4 lu,
                                         int64_t s) {
    if (it < 0) return;
    const float inv = 1.f / (v.dt * m);
    l.beta[s] = make_float4(lu.x * inv, lu.y * inv, lu.z * inv, kappa_of(v, kind, it)[s]);
}

template <int DIM>
__device__ __forceinline__ void adj_in_item(const SlotView &v, const Lam &l, const float *gx, const float *gv, int kp,
                                            int64_t s) {
    const int64_t b = (int64_t)v.perm[s] * DIM;
    const float x0 = gx[b], x1 = gx[b + 1], x2 = DIM == 3 ? gx[b + 2] : 0.f;
    const float v0 = gv[b], v1 = gv[b + 1], v2 = DIM == 3 ? gv[b + 2] : 0.f;
    l.x[s] = make_float4(x0, x1, x2, 0.f);
    // x' = x + v' dt: the step's velocity output also moved the positions
    const float4 lu = make_float4(v0 + v.dt * x0, v1 + v.dt * x1, v2 + v.dt * x2, v.rho0[s]);
    l.u[s] = lu;
    put_beta(v, l, kSolveDens, kp - 1, v.pos[s].w, lu, s);
    l.psi[s] = 0.f;
    l.alpha[s] = 0.f;
}

// Reverse of the velocity update of iteration `it`.
template <int TPP>
__device__ __forceinline__ void adj_kappa_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int kind,
                                               int it, int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float4 pi = v.pos[i];
    const float mi = pi.w;
    const float4 bi = l.beta[i];
    const float ki = bi.w;
    const float bx = bi.x, by = bi.y, bz = bi.z;
    float lk = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    for_pairs(v, ln, s,
        [&](int j) {
            const float4 pj = v.pos[j];
            const Pair P(v, pi, pj);
            const float4 bj = l.beta[j];
            const float dx = bx - bj.x, dy = by - bj.y, dz = bz - bj.z;
            const float rd = P.dot(dx, dy, dz);
            lk -= pj.w * P.g * rd;
            const float cK = ki * pj.w + bj.w * mi;
            gx -= cK * (P.g * dx + P.G2 * rd * P.x);
            gy -= cK * (P.g * dy + P.G2 * rd * P.y);
            gz -= cK * (P.g * dz + P.G2 * rd * P.z);
        },
        [&](int b) {
            const float4 pb = v.bpos[b];
            const Pair P(v, pi, pb);
            const float rd = P.dot(bx, by, bz);
            lk -= pb.w * P.g * rd;
            const float cK = ki * pb.w;
            gx -= cK * (P.g * bx + P.G2 * rd * P.x);
            gy -= cK * (P.g * by + P.G2 * rd * P.y);
            gz -= cK * (P.g * bz + P.G2 * rd * P.z);
        });
    lk = ln.sum(lk);
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    if (s >= v.n || ln.q != 0) return;
    const float alpha = v.mpsi[s].w;
    const float lsi = ki > 0.f ? lk / alpha : 0.f;
    l.alpha[s] -= lk * ki / alpha;
    l.psi[s] += lsi;
    const float4 u = v.u[((int64_t)kind * v.max_iters + it) * v.cap + s];
    l.us[s] = make_float4(u.x, u.y, u.z, lsi);
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + gx, o.y + gy, o.z + gz, 0.f);
}

// Reverse of the divergence of iteration `it`.
template <int TPP>
__device__ __forceinline__ void adj_vel_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int kind, int it,
                                             int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float4 pi = v.pos[i];
    const float mi = pi.w;
    const float4 ui = l.us[i];
    const float lsi = ui.w;
    float ax = 0.f, ay = 0.f, az = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    auto term = [&](const Pair &P, float cS, float4 uj) {
        ax += cS * P.g * P.x;
        ay += cS * P.g * P.y;
        az += cS * P.g * P.z;
        const float dx = ui.x - uj.x, dy = ui.y - uj.y, dz = ui.z - uj.z;
        const float rd = P.dot(dx, dy, dz);
        gx += cS * (P.g * dx + P.G2 * rd * P.x);
        gy += cS * (P.g * dy + P.G2 * rd * P.y);
        gz += cS * (P.g * dz + P.G2 * rd * P.z);
    };
    for_pairs(v, ln, s,
        [&](int j) {
            const float4 pj = v.pos[j];
            const float4 uj = l.us[j];
            term(Pair(v, pi, pj), lsi * pj.w + uj.w * mi, uj);
        },
        [&](int b) {
            const float4 pb = v.bpos[b];
            term(Pair(v, pi, pb), lsi * pb.w, v.bvel[b]);
        });
    ax = ln.sum(ax);
    ay = ln.sum(ay);
    az = ln.sum(az);
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    if (s >= v.n || ln.q != 0) return;
    const float4 lu = l.u[s];
    const float4 nu = make_float4(lu.x + v.dt * ax, lu.y + v.dt * ay, lu.z + v.dt * az, lu.w);
    l.u[s] = nu;
    put_beta(v, l, kind, it - 1, mi, nu, s);
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + v.dt * gx, o.y + v.dt * gy, o.z + v.dt * gz, 0.f);
}

// Reverse of u0 = v + dt (g + mu V): lam_v = lam_u0 + (dV/dv)^T lam_a with
// lam_a = dt lam_u0; also lam_x, lam_psi and dL/dmu = sum_i lam_a_i . V_i.
// Returns the particle's share of dL/dmu.
template <int DIM, int TPP>
__device__ __forceinline__ double adj_visc_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int kd,
                                                int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float lap = 2.f * (2.f + DIM);
    const float4 pi = v.pos[i];
    const float mi = pi.w;
    const float4 lui = l.u[i];
    const float lax = v.dt * lui.x, lay = v.dt * lui.y, laz = v.dt * lui.z;
    const float4 vi = v.vmid[i];  // w: psi
    const float psii = vi.w, r0i = lui.w;
    float avx = 0.f, avy = 0.f, avz = 0.f, gx = 0.f, gy = 0.f, gz = 0.f, lp = 0.f;
    float Vx = 0.f, Vy = 0.f, Vz = 0.f;
    for_pairs(v, ln, s,
        [&](int j) {
            const float4 pj = v.pos[j];
            const Pair P(v, pi, pj);
            const float den = v.eps + P.r2;
            const float phi = P.g / den;
            const float dphi = P.G2 / den - 2.f * P.g / (den * den);
            const float4 vj = v.vmid[j];
            const float4 luj = l.u[j];
            const float psij = vj.w, r0j = luj.w;
            const float ljx = v.dt * luj.x, ljy = v.dt * luj.y, ljz = v.dt * luj.z;
            const float wx = vi.x - vj.x, wy = vi.y - vj.y, wz = vi.z - vj.z;
            const float vr = P.dot(wx, wy, wz);
            const float ci = v.mu * lap * pj.w / (r0i * psij);
            const float cj = v.mu * lap * mi / (r0j * psii);
            const float rli = P.dot(lax, lay, laz), rlj = P.dot(ljx, ljy, ljz);
            const float fv = (ci * rli - cj * rlj) * phi;
            avx += fv * P.x;
            avy += fv * P.y;
            avz += fv * P.z;
            lp += cj * phi * vr * rlj / psii;
            const float ti = vr * rli * dphi, tj = vr * rlj * dphi;
            gx += ci * (phi * (rli * wx + vr * lax) + ti * P.x) - cj * (phi * (rlj * wx + vr * ljx) + tj * P.x);
            gy += ci * (phi * (rli * wy + vr * lay) + ti * P.y) - cj * (phi * (rlj * wy + vr * ljy) + tj * P.y);
            gz += ci * (phi * (rli * wz + vr * laz) + ti * P.z) - cj * (phi * (rlj * wz + vr * ljz) + tj * P.z);
            const float fV = lap * (pj.w / psij) * phi * vr;
            Vx += fV * P.x;
            Vy += fV * P.y;
            Vz += fV * P.z;
        },
        [&](int) {});
    avx = ln.sum(avx);
    avy = ln.sum(avy);
    avz = ln.sum(avz);
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    lp = ln.sum(lp);
    Vx = ln.sum(Vx);
    Vy = ln.sum(Vy);
    Vz = ln.sum(Vz);
    if (s >= v.n || ln.q != 0) return 0.0;
    const float4 nu = make_float4(lui.x + avx, lui.y + avy, lui.z + avz, lui.w);
    l.u2[s] = nu;
    put_beta(v, l, kSolveDiv, kd - 1, mi, nu, s);
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + gx, o.y + gy, o.z + gz, 0.f);
    l.psi[s] += lp;
    return (double)((lax * Vx + lay * Vy + laz * Vz) / r0i);
}

// Surface tension, first reverse sweep, over the template candidates the
// forward visits (sph.py:156-166).  With c_ij = 2 psi0_i / (psi_i + psi_j),
// B_ij = -gamma m_j C(r) r_ij / r + gamma (n_i - n_j) and lam_a = dt lam_u:
//   lam_n_i    = gamma sum_j (c_ij lam_a_i - c_ji lam_a_j),
//   lam_psi_i -= sum_j (c_ij lam_a_i.B_ij + c_ji lam_a_j.B_ji) / (psi_i + psi_j),
//   lam_x_i   += sum_j (k_ij D_C(lam_a_i) - k_ji D_C(lam_a_j)), k_ij = -gamma m_j c_ij,
// D_C(w) = (C/r) w + ((C' - C/r) / r^2)(r_ij.w) r_ij.  Pairs count only where
// both particles' phase-0 volume fraction exceeds 0.99, as in the forward.
template <int DIM, int TPP>
__device__ __forceinline__ void adj_st1_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float4 pi = v.pos[i];
    const float4 mpi = v.mpsi[i];
    const float mi = mpi.x, psii = mpi.y, r0i = mpi.z;
    const float4 ni = v.nrm[i];
    const float4 lui = l.u[i];
    const float lax = v.dt * lui.x, lay = v.dt * lui.y, laz = v.dt * lui.z;
    const float gam = v.gamma;
    float nx = 0.f, ny = 0.f, nz = 0.f, lp = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    bool ok;
    const long long code = cell_code<DIM>(pi, v.geo, ok);
    if (s < v.n && ok && v.vf0[i] > 0.99f) {
        visit_candidates<DIM, TPP>(v.start, v.geo, code, 0, ln.q, [&](int j) {
            const float4 pj = v.pos[j];
            const float x = pi.x - pj.x, y = pi.y - pj.y, z = pi.z - pj.z;
            const float r2 = x * x + y * y + z * z;
            if (!(r2 > 0.f) || !(v.vf0[j] > 0.99f)) return;
            float r;
            const float ri = pair_rinv(r2, r);
            const float q = r * v.inv_h;
            const float gC = kcoh(q) * v.c_coh * ri;
            const float G2C = (kcohd(q) * v.c_coh * v.inv_h - gC) * (ri * ri);
            const float4 mpj = v.mpsi[j];
            const float mj = mpj.x, psij = mpj.y, r0j = mpj.z;
            const float4 nj = v.nrm[j];
            const float4 luj = l.u[j];
            const float ljx = v.dt * luj.x, ljy = v.dt * luj.y, ljz = v.dt * luj.z;
            const float sum = psii + psij;
            const float cij = 2.f * r0i / sum, cji = 2.f * r0j / sum;
            const float dnx = ni.x - nj.x, dny = ni.y - nj.y, dnz = ni.z - nj.z;
            const float rli = x * lax + y * lay + z * laz, rlj = x * ljx + y * ljy + z * ljz;
            const float laBij = -gam * mj * gC * rli + gam * (dnx * lax + dny * lay + dnz * laz);
            const float laBji = gam * mi * gC * rlj - gam * (dnx * ljx + dny * ljy + dnz * ljz);
            nx += gam * (cij * lax - cji * ljx);
            ny += gam * (cij * lay - cji * ljy);
            nz += gam * (cij * laz - cji * ljz);
            lp -= (cij * laBij + cji * laBji) / sum;
            const float kij = -gam * mj * cij, kji = -gam * mi * cji;
            gx += kij * (gC * lax + G2C * rli * x) - kji * (gC * ljx + G2C * rlj * x);
            gy += kij * (gC * lay + G2C * rli * y) - kji * (gC * ljy + G2C * rlj * y);
            gz += kij * (gC * laz + G2C * rli * z) - kji * (gC * ljz + G2C * rlj * z);
        });
    }
    nx = ln.sum(nx);
    ny = ln.sum(ny);
    nz = ln.sum(nz);
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    lp = ln.sum(lp);
    if (s >= v.n || ln.q != 0) return;
    l.n[s] = make_float4(nx, ny, nz, 0.f);
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + gx, o.y + gy, o.z + gz, 0.f);
    l.psi[s] += lp;
}

// Surface tension, second reverse sweep: the normals n_i = h sum_j -(X_j /
// psi_j) g_ij r_ij over the pairs within h,
//   lam_x_i   += h sum_j ((X_i / psi_i) D(lam_n_j) - (X_j / psi_j) D(lam_n_i)),
//   lam_psi_i -= h (X_i / psi_i^2) sum_j g_ij r_ij.lam_n_j,
// D(w) = g w + G2 (r_ij.w) r_ij.
template <int TPP>
__device__ __forceinline__ void adj_st2_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float4 pi = v.pos[i];
    const float psii = v.mpsi[i].y;
    const float ai = pi.w / psii;
    const float4 ni = l.n[i];
    float gx = 0.f, gy = 0.f, gz = 0.f, lp = 0.f;
    for_pairs(v, ln, s,
        [&](int j) {
            const float4 pj = v.pos[j];
            const Pair P(v, pi, pj);
            const float aj = pj.w / v.mpsi[j].y;
            const float4 nj = l.n[j];
            const float rj = P.dot(nj.x, nj.y, nj.z), rI = P.dot(ni.x, ni.y, ni.z);
            gx += ai * (P.g * nj.x + P.G2 * rj * P.x) - aj * (P.g * ni.x + P.G2 * rI * P.x);
            gy += ai * (P.g * nj.y + P.G2 * rj * P.y) - aj * (P.g * ni.y + P.G2 * rI * P.y);
            gz += ai * (P.g * nj.z + P.G2 * rj * P.z) - aj * (P.g * ni.z + P.G2 * rI * P.z);
            lp += P.g * rj;
        },
        [&](int) {});
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    lp = ln.sum(lp);
    if (s >= v.n || ln.q != 0) return;
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + v.h * gx, o.y + v.h * gy, o.z + v.h * gz, 0.f);
    l.psi[s] -= v.h * ai / psii * lp;
}

// lam of alpha's two sums: (lam_alpha1 xyz, lam_alpha2) where alpha was not clamped.
__device__ __forceinline__ void adj_alpha_item(const SlotView &v, const Lam &l, int64_t s) {
    const float4 a1 = v.a1[s];
    const float m = v.mpsi[s].x;
    const float raw = (a1.x * a1.x + a1.y * a1.y + a1.z * a1.z) / m + v.a2[s];
    const bool on = !(raw < 1e-4f);
    const float la = on ? l.alpha[s] : 0.f;
    const float f = la * 2.f / m;
    l.a1[s] = make_float4(f * a1.x, f * a1.y, f * a1.z, la);
}

// Reverse of rho_i = sum_j m_j W_ij, alpha1_i = sum_j X_j g r_ij and
// alpha2_i = sum_j (X_j^2 / m_j) W'(r)^2 (X = m for DFSPH): position terms only.
template <int TPP>
__device__ __forceinline__ void adj_density_item(const SlotView &v, const Lam &l, const Lanes<TPP> &ln, int64_t s) {
    const int64_t i = s < v.n ? s : 0;  // (lanes past the end compute and drop)
    const float4 pi = v.pos[i];
    const float mi = pi.w;
    const float lpi = l.psi[i];
    const float4 ai = l.a1[i];
    float gx = 0.f, gy = 0.f, gz = 0.f;
    for_pairs(v, ln, s,
        [&](int j) {
            const float4 pj = v.pos[j];
            const Pair P(v, pi, pj);
            const float4 aj = l.a1[j];
            const float ri = P.dot(ai.x, ai.y, ai.z), rj = P.dot(aj.x, aj.y, aj.z);
            const float cR = (lpi * pj.w + l.psi[j] * mi) * P.g + (ai.w * pj.w + aj.w * mi) * 2.f * P.g * P.W2;
            const float cA = P.G2 * (pj.w * ri - mi * rj);
            gx += cR * P.x + P.g * (pj.w * ai.x - mi * aj.x) + cA * P.x;
            gy += cR * P.y + P.g * (pj.w * ai.y - mi * aj.y) + cA * P.y;
            gz += cR * P.z + P.g * (pj.w * ai.z - mi * aj.z) + cA * P.z;
        },
        [&](int b) {
            const float4 pb = v.bpos[b];
            const Pair P(v, pi, pb);
            const float ri = P.dot(ai.x, ai.y, ai.z);
            const float c = lpi * pb.w * P.g + pb.w * P.G2 * ri;
            gx += c * P.x + pb.w * P.g * ai.x;
            gy += c * P.y + pb.w * P.g * ai.y;
            gz += c * P.z + pb.w * P.g * ai.z;
        });
    gx = ln.sum(gx);
    gy = ln.sum(gy);
    gz = ln.sum(gz);
    if (s >= v.n || ln.q != 0) return;
    const float4 o = l.x[s];
    l.x[s] = make_float4(o.x + gx, o.y + gy, o.z + gz, 0.f);
}

template <int DIM>
__device__ __forceinline__ void adj_out_item(const SlotView &v, const float4 *lx, const float4 *lu, float *gx,
                                             float *gv, int accumulate, int64_t s) {
    const int64_t b = (int64_t)v.perm[s] * DIM;
    const float4 x = lx[s];
    const float xv[3] = {x.x, x.y, x.z};
#pragma unroll
    for (int d = 0; d < DIM; ++d) gx[b + d] = accumulate ? gx[b + d] + xv[d] : xv[d];
    if (gv) {
        const float4 u = lu[s];
        const float uv[3] = {u.x, u.y, u.z};
#pragma unroll
        for (int d = 0; d < DIM; ++d) gv[b + d] = uv[d];
    }
}

// ----------------------------------------------------------------------------- one kernel a sweep
// The sweeps as separate launches, where the cooperative kernel is not taken.
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_adj_in(SlotView v, Lam l, const float *__restrict__ gx,
                                                   const float *__restrict__ gv, int kp) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < v.n) adj_in_item<DIM>(v, l, gx, gv, kp, s);
}

__global__ void __launch_bounds__(kBlock) k_adj_kappa(SlotView v, Lam l, int kind, int it) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    adj_kappa_item<1>(v, l, Lanes<1>(), kind, it, s);
}

__global__ void __launch_bounds__(kBlock) k_adj_vel(SlotView v, Lam l, int kind, int it) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    adj_vel_item<1>(v, l, Lanes<1>(), kind, it, s);
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_adj_visc(SlotView v, Lam l, int kd, double *partials,
                                                     unsigned int *ticket, double *gmu) {
    __shared__ double sh[kBlock / 32];
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const double contrib = adj_visc_item<DIM, 1>(v, l, Lanes<1>(), kd, s);
    const double bs = block_sum<kBlock>(contrib, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (last_block_done(ticket, gridDim.x)) {
        double a = 0.0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += kBlock) a += __ldcg(partials + i);
        a = block_sum<kBlock>(a, sh);
        if (threadIdx.x == 0) {
            *gmu += a;
            *ticket = 0;
        }
    }
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_adj_st1(SlotView v, Lam l) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    adj_st1_item<DIM, 1>(v, l, Lanes<1>(), s);
}

__global__ void __launch_bounds__(kBlock) k_adj_st2(SlotView v, Lam l) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    adj_st2_item<1>(v, l, Lanes<1>(), s);
}

__global__ void __launch_bounds__(kBlock) k_adj_alpha(SlotView v, Lam l) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < v.n) adj_alpha_item(v, l, s);
}

__global__ void __launch_bounds__(kBlock) k_adj_density(SlotView v, Lam l) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    adj_density_item<1>(v, l, Lanes<1>(), s);
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_adj_out(SlotView v, const float4 *__restrict__ lx,
                                                    const float4 *__restrict__ lu, float *gx, float *gv,
                                                    int accumulate) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < v.n) adj_out_item<DIM>(v, lx, lu, gx, gv, accumulate, s);
}

// ----------------------------------------------------------------------------- one launch a substep
struct AdjArgs {
    const float *gx_out, *gv_out;
    float *gx_in, *gv_in;
    double *gmu, *sums;  // sums: 32 per block, one per warp
    unsigned int *bar;
    ScenePersist *sp, *host_sp;  // what a reverse that gives up marks; its pinned copy
    unsigned int absent;         // blocks that will not come (GridBarrier)
    int kd, kp;
};

// The reverse of a substep in one cooperative launch: fourteen or more sweeps of a
// few microseconds each are otherwise as many launches.  A block's particles
// in runs of 32 as elsewhere; with TPP lanes per particle a run takes TPP warps.
template <int DIM, int TPP>
__global__ void __launch_bounds__(1024, 1) k_adj_step(const __grid_constant__ SlotView v,
                                                      const __grid_constant__ Lam lam,
                                                      const __grid_constant__ AdjArgs a) {
    __shared__ double sh[kBlock / 32];
    GridBarrier bar{a.bar, a.absent};
    Lam l = lam;
    // item(slot) for every lane of the particles' lane groups; all lanes of a warp call
    auto sweep = [&](auto &&item) {
        const WarpShare w(v.n);
        const Lanes<TPP> ln;
        for (int64_t i = threadIdx.x >> 5; i < (int64_t)w.runs * TPP; i += blockDim.x >> 5)
            item(ln, ((int64_t)w.first * TPP + i) * ln.PPW + ln.p);
    };
    auto own = [&](const Lanes<TPP> &ln, int64_t s) { return s < v.n && ln.q == 0; };
    auto solve = [&](int kind, int iters) {
        for (int it = iters - 1; it >= 0; --it) {
            sweep([&](const Lanes<TPP> &ln, int64_t s) { adj_kappa_item<TPP>(v, l, ln, kind, it, s); });
            if (!bar.sync()) return false;
            sweep([&](const Lanes<TPP> &ln, int64_t s) {
                adj_vel_item<TPP>(v, l, ln, kind, it, s);
                // lam_alpha is complete after the last kappa sweep
                if (kind == kSolveDiv && it == 0 && own(ln, s)) adj_alpha_item(v, l, s);
            });
            if (!bar.sync()) return false;
        }
        return true;
    };
    auto run = [&]() {
        sweep([&](const Lanes<TPP> &ln, int64_t s) {
            if (own(ln, s)) adj_in_item<DIM>(v, l, a.gx_out, a.gv_out, a.kp, s);
        });
        if (!bar.sync() || !solve(kSolveDens, a.kp)) return false;
        double g = 0.0;  // this lane's particles' share of dL/dmu
        sweep([&](const Lanes<TPP> &ln, int64_t s) {
            g += adj_visc_item<DIM, TPP>(v, l, ln, a.kd, s);
            // the surface tension's reverse reads the same lam_a = dt lam_u
            if (v.gamma != 0.f) adj_st1_item<DIM, TPP>(v, l, ln, s);
            if (a.kd == 0 && own(ln, s)) adj_alpha_item(v, l, s);
        });
        g = warp_sum(g);
        if ((threadIdx.x & 31) == 0) a.sums[blockIdx.x * 32 + (threadIdx.x >> 5)] = g;
        if (!bar.sync()) return false;
        if (v.gamma != 0.f) {
            sweep([&](const Lanes<TPP> &ln, int64_t s) { adj_st2_item<TPP>(v, l, ln, s); });
            if (a.kd == 0 && !bar.sync()) return false;
        }
        float4 *u = l.u;
        l.u = l.u2;
        l.u2 = u;
        if (!solve(kSolveDiv, a.kd)) return false;
        sweep([&](const Lanes<TPP> &ln, int64_t s) {
            adj_density_item<TPP>(v, l, ln, s);
            if (own(ln, s)) adj_out_item<DIM>(v, l.x, l.u, a.gx_in, a.gv_in, 0, s);
        });
        return true;
    };
    const bool done = run();
    if (!last_block_done(a.bar + kBarLeft, gridDim.x)) return;
    // A barrier given up (by any block, whatever this one saw) leaves the gradients
    // unfinished: they all become NaN, and the next reading of the scalars fails.
    const unsigned int given_up = __ldcg(a.bar + kBarGaveUp);
    // dL/dmu: the warps' sums, in a fixed order
    double g = 0.0;
    const int warps = blockDim.x >> 5;
    for (int i = threadIdx.x; i < (int)gridDim.x * warps && threadIdx.x < kBlock; i += kBlock)
        g += __ldcg(a.sums + i / warps * 32 + i % warps);
    g = coop_sum256(g, sh);
    const bool ok = done && !given_up;
    if (!ok)
        for (int64_t i = threadIdx.x; i < (int64_t)v.n * DIM; i += blockDim.x)
            a.gx_in[i] = a.gv_in[i] = __int_as_float(0x7fffffff);
    if (threadIdx.x != 0) return;
    *a.gmu += ok ? g : __longlong_as_double(0x7ff8000000000000ll);
    if (!ok) a.sp->gave_up = a.host_sp->gave_up = 1;
    a.bar[kBarCount] = a.bar[kBarGaveUp] = a.bar[kBarLeft] = 0;
}

__global__ void __launch_bounds__(kBlock) k_adj_in_density(SlotView v, Lam l, const float *__restrict__ grho) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s >= v.n) return;
    l.psi[s] = grho[v.perm[s]];
    l.a1[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    l.x[s] = make_float4(0.f, 0.f, 0.f, 0.f);
}

int fail_text(int code, const char *msg) {
    set_last_error_text(msg);
    return code;
}

SlotView slot_view(const tsph_tape &t, int slot) {
    const TapeArrays &a = t.a;
    const TapeMeta &m = t.host_meta[slot];
    const SceneConst &c = t.ctx->k.s0;
    SlotView v;
    const int64_t o = (int64_t)slot * a.cap;
    v.perm = a.perm + o;
    v.pos = a.pos + o;
    v.mpsi = a.mpsi + o;
    v.a1 = a.a1 + o;
    v.vmid = a.vmid + o;
    v.a2 = a.a2 + o;
    v.rho0 = a.rho0 + o;
    v.cnt = a.cnt + o;
    v.nbr = a.nbr + (int64_t)slot * a.nbr_max * a.cap;
    v.bpos = a.bpos + (int64_t)slot * a.bcap;
    v.bvel = a.bvel + (int64_t)slot * a.bcap;
    v.u = a.u + (int64_t)slot * 2 * a.max_iters * a.cap;
    v.kap = a.kap + (int64_t)slot * 2 * a.max_iters * a.cap;
    v.cap = a.cap;
    v.n = m.n;
    v.max_iters = a.max_iters;
    v.dt = m.dt;
    v.mu = m.mu;
    v.h = c.h;
    v.h2 = c.h2;
    v.inv_h = c.inv_h;
    v.sig_h = c.sig_h;
    v.eps = 0.01f * c.h2;
    v.gamma = a.nrm ? c.gamma : 0.f;
    v.c_coh = c.c_coh;
    v.nrm = a.nrm ? a.nrm + o : nullptr;
    v.vf0 = a.vf0 ? a.vf0 + o : nullptr;
    v.start = a.start ? a.start + (int64_t)slot * a.nstart : nullptr;
    Geo &g = v.geo;
    for (int d = 0; d < 3; ++d) g.lb[d] = c.lb[d];
    g.h = c.h;
    g.h2 = c.h2;
    g.inv_h = c.inv_h;
    g.sig = c.sig;
    g.sig_h = c.sig_h;
    g.node_num = c.node_num;
    g.nx = c.nx;
    g.nxny = c.nxny;
    g.cbase = c.cbase;
    g.R = t.ctx->k.R;
    g.row_trim = c.row_trim;
    return v;
}

Lam lam_of(const tsph_tape &t) {
    return {t.lam_u, t.lam_u2, t.lam_x, t.lam_beta, t.lam_us, t.lam_a1, t.lam_n, t.lam_psi, t.lam_alpha};
}

// Up to this many warps of fluid particles per SM a substep is reversed in one
// launch.  (The forward step's limit, which counts the boundary's warps too; its other
// conditions do not matter to the reverse, which reads the tape alone.)
constexpr int64_t kAdjWarpsPerSm = 512;

// Eight lanes per particle while the SMs' 32 warps hold them all, then four, then
// one: the sweeps of a small scene are chains of list blocks and their gathers,
// one after another in a lane (a rollout of 2,028 particles: 5.1 ms, 6.5 with one lane).
template <int DIM>
cudaError_t launch_adj_step(tsph_ctx &c, const SlotView &v, const Lam &l, const AdjArgs &a, cudaStream_t st) {
    const int64_t warps = ((int64_t)v.n + 31) / 32, runs = (warps + c.sms - 1) / c.sms;
    if (runs * 8 <= 32) return launch_coop(k_adj_step<DIM, 8>, c.sms, coop_threads(runs * 8 * c.sms, c.sms), st, v, l, a);
    if (runs * 4 <= 32) return launch_coop(k_adj_step<DIM, 4>, c.sms, coop_threads(runs * 4 * c.sms, c.sms), st, v, l, a);
    return launch_coop(k_adj_step<DIM, 1>, c.sms, coop_threads(warps, c.sms), st, v, l, a);
}

// Host copy of every slot's metadata (one synchronisation per recording).
int sync_meta(tsph_tape &t, cudaStream_t st) {
    if (t.host_valid) return TSPH_OK;
    cudaError_t e = cudaMemcpyAsync(t.host_meta, t.a.meta, sizeof(TapeMeta) * t.a.slots, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail_text(TSPH_ERR_CUDA, cudaGetErrorString(e));
    t.host_valid = 1;
    return TSPH_OK;
}

int check_slot(tsph_ctx *c, tsph_tape *t, int slot) {
    if (!c || !t || t->ctx != c) return fail_text(TSPH_ERR_INVALID, "tape does not belong to this context");
    if (slot < 0 || slot >= t->a.slots) return fail_text(TSPH_ERR_INVALID, "tape slot out of range");
    return TSPH_OK;
}

int usable(const tsph_tape &t, int slot) {
    const TapeMeta &m = t.host_meta[slot];
    if (m.status) {
        char buf[160];
        std::snprintf(buf, sizeof(buf), "tape slot %d cannot be reversed (TSPH_TAPE_* bits 0x%x)", slot, m.status);
        return fail_text(TSPH_ERR_STATE, buf);
    }
    if (m.n <= 0) return fail_text(TSPH_ERR_STATE, "tape slot holds no recording");
    return TSPH_OK;
}

}  // namespace

void launch_tape_state(tsph_ctx &c, cudaStream_t st) {
    const int64_t n = c.F.cap > c.B.cap ? c.F.cap : c.B.cap;
    c.launches += 1;
    k_tape_state<<<blocks_for(n), kBlock, 0, st>>>(c.k, c.F, c.B, c.rec_tape->a);
    const TapeArrays &a = c.rec_tape->a;
    if (a.start) {
        c.launches += 1;
        k_tape_start<<<blocks_for(a.nstart), kBlock, 0, st>>>(c.F, a);
    }
}

void launch_tape_iter(tsph_ctx &c, int kind, cudaStream_t st) {
    c.launches += 1;
    k_tape_iter<<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.k, c.F, kind, c.rec_tape->a);
}

void launch_tape_vmid(tsph_ctx &c, cudaStream_t st) {
    c.launches += 1;
    k_tape_vmid<<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.k, c.F, c.rec_tape->a);
}

void launch_tape_end(tsph_ctx &c, cudaStream_t st) {
    c.launches += 1;
    k_tape_end<<<1, 1, 0, st>>>(c.k, c.rec_tape->a);
}

int tape_begin(tsph_tape &t, int slot, cudaStream_t st) {
    k_tape_begin<<<1, 1, 0, st>>>(t.a, slot);
    t.host_valid = 0;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TSPH_OK : fail_text(TSPH_ERR_CUDA, cudaGetErrorString(e));
}

void launch_density_out(tsph_ctx &c, float *out, cudaStream_t st) {
    k_density_out<<<blocks_for(c.F.cap), kBlock, 0, st>>>(c.k, c.F, out);
}

}  // namespace tsph

using namespace tsph;

extern "C" {

int tsph_tape_create(tsph_ctx *c, int slots, int max_iters, tsph_tape **out) {
    if (!c || !out || slots < 1 || max_iters < 1) return fail_text(TSPH_ERR_INVALID, "bad argument");
    *out = nullptr;
    if (c->n_scenes != 1 || c->batch) return fail_text(TSPH_ERR_INVALID, "the adjoint supports one-scene contexts");
    if (c->p.solver_type != TSPH_DFSPH || c->p.fbm_enabled)
        return fail_text(TSPH_ERR_INVALID, "the adjoint supports DFSPH without the volume-fraction update");
    tsph_tape *t = new (std::nothrow) tsph_tape();
    if (!t) return fail_text(TSPH_ERR_INVALID, "out of host memory");
    t->ctx = c;
    TapeArrays &a = t->a;
    a.cap = c->F.cap;
    a.bcap = c->B.cap;
    a.slots = slots;
    a.max_iters = max_iters;
    a.nbr_max = c->k.nbr_max;
    cudaError_t err = cudaSuccess;
    auto get = [&](size_t bytes) -> void * {
        void *p = nullptr;
        if (err != cudaSuccess) return nullptr;
        err = cudaMalloc(&p, bytes < 16 ? 16 : bytes);
        if (err != cudaSuccess) return nullptr;
        err = cudaMemset(p, 0, bytes < 16 ? 16 : bytes);
        t->allocs.push_back(p);
        return p;
    };
    const size_t S = (size_t)slots, N = (size_t)a.cap, NB = (size_t)a.bcap;
    a.perm = (int *)get(S * N * sizeof(int));
    a.pos = (float4 *)get(S * N * sizeof(float4));
    a.mpsi = (float4 *)get(S * N * sizeof(float4));
    a.a1 = (float4 *)get(S * N * sizeof(float4));
    a.vmid = (float4 *)get(S * N * sizeof(float4));
    a.a2 = (float *)get(S * N * sizeof(float));
    a.rho0 = (float *)get(S * N * sizeof(float));
    a.cnt = (unsigned int *)get(S * N * sizeof(unsigned int));
    a.nbr = (int *)get(S * (size_t)a.nbr_max * N * sizeof(int));
    a.u = (float4 *)get(S * 2 * (size_t)max_iters * N * sizeof(float4));
    a.kap = (float *)get(S * 2 * (size_t)max_iters * N * sizeof(float));
    a.bpos = (float4 *)get(S * NB * sizeof(float4));
    a.bvel = (float4 *)get(S * NB * sizeof(float4));
    a.meta = (TapeMeta *)get(S * sizeof(TapeMeta));
    a.dslot = (int *)get(sizeof(int));
    t->lam_u = (float4 *)get(N * sizeof(float4));
    t->lam_u2 = (float4 *)get(N * sizeof(float4));
    t->lam_x = (float4 *)get(N * sizeof(float4));
    t->lam_a1 = (float4 *)get(N * sizeof(float4));
    t->lam_beta = (float4 *)get(N * sizeof(float4));
    t->lam_us = (float4 *)get(N * sizeof(float4));
    t->lam_psi = (float *)get(N * sizeof(float));
    t->lam_alpha = (float *)get(N * sizeof(float));
    t->partials = (double *)get(std::max(N / kBlock + 2, (size_t)c->sms * 32) * sizeof(double));
    t->bar = (unsigned int *)get(kBarWords * sizeof(unsigned int));
    t->ticket = (unsigned int *)get(sizeof(unsigned int));
    if (c->st_on) {
        a.nstart = c->k.total_nodes + 1;
        a.nrm = (float4 *)get(S * N * sizeof(float4));
        a.vf0 = (float *)get(S * N * sizeof(float));
        a.start = (int *)get(S * (size_t)a.nstart * sizeof(int));
        t->lam_n = (float4 *)get(N * sizeof(float4));
    }
    if (err == cudaSuccess) err = cudaMallocHost((void **)&t->host_meta, S * sizeof(TapeMeta));
    if (err == cudaSuccess) err = cudaDeviceSynchronize();
    if (err != cudaSuccess) {
        tsph_tape_destroy(t);
        return fail_text(TSPH_ERR_CUDA, cudaGetErrorString(err));
    }
    *out = t;
    return TSPH_OK;
}

int tsph_tape_destroy(tsph_tape *t) {
    if (!t) return TSPH_OK;
    // the context only points at a tape during a recorded call, so it need not be touched
    for (void *p : t->allocs) cudaFree(p);
    if (t->host_meta) cudaFreeHost(t->host_meta);
    delete t;
    return TSPH_OK;
}

int tsph_substep_adjoint(tsph_ctx *c, tsph_tape *t, int slot, const float *gx_out, const float *gv_out,
                         float *gx_in, float *gv_in, double *gmu, void *stream) {
    int rc = check_slot(c, t, slot);
    if (rc) return rc;
    if (!gx_out || !gv_out || !gx_in || !gv_in || !gmu) return fail_text(TSPH_ERR_INVALID, "null gradient pointer");
    cudaStream_t st = (cudaStream_t)stream;
    rc = sync_meta(*t, st);
    if (rc) return rc;
    rc = usable(*t, slot);
    if (rc) return rc;
    const TapeMeta &m = t->host_meta[slot];
    if (m.kd > t->a.max_iters || m.kp > t->a.max_iters)
        return fail_text(TSPH_ERR_STATE, "tape slot ran more iterations than it holds");
    const SlotView v = slot_view(*t, slot);
    const int nb = blocks_for(v.n);
    Lam l = lam_of(*t);
    if (c->use_graph && c->sms && ((int64_t)v.n + 31) / 32 <= kAdjWarpsPerSm * c->sms) {
        const AdjArgs a = {gx_out, gv_out, gx_in, gv_in, gmu, t->partials, t->bar,
                           c->k.sp, c->host_sp, c->absent, m.kd, m.kp};
        const cudaError_t e = c->k.dim == 3 ? launch_adj_step<3>(*c, v, l, a, st) : launch_adj_step<2>(*c, v, l, a, st);
        if (e == cudaSuccess) return TSPH_OK;
        // this process may not use every SM at once: separate launches
        if (e != cudaErrorCooperativeLaunchTooLarge) return fail_text(TSPH_ERR_CUDA, cudaGetErrorString(e));
        (void)cudaGetLastError();
    }
    auto solve = [&](int kind, int iters) {
        for (int it = iters - 1; it >= 0; --it) {
            k_adj_kappa<<<nb, kBlock, 0, st>>>(v, l, kind, it);
            k_adj_vel<<<nb, kBlock, 0, st>>>(v, l, kind, it);
        }
    };
    const bool d3 = c->k.dim == 3;
    if (d3) k_adj_in<3><<<nb, kBlock, 0, st>>>(v, l, gx_out, gv_out, m.kp);
    else k_adj_in<2><<<nb, kBlock, 0, st>>>(v, l, gx_out, gv_out, m.kp);
    solve(kSolveDens, m.kp);
    if (d3) k_adj_visc<3><<<nb, kBlock, 0, st>>>(v, l, m.kd, t->partials, t->ticket, gmu);
    else k_adj_visc<2><<<nb, kBlock, 0, st>>>(v, l, m.kd, t->partials, t->ticket, gmu);
    if (v.gamma != 0.f) {
        // the surface tension's reverse reads the same lam_a = dt lam_u as k_adj_visc
        if (d3) k_adj_st1<3><<<nb, kBlock, 0, st>>>(v, l);
        else k_adj_st1<2><<<nb, kBlock, 0, st>>>(v, l);
        k_adj_st2<<<nb, kBlock, 0, st>>>(v, l);
    }
    std::swap(l.u, l.u2);
    solve(kSolveDiv, m.kd);
    k_adj_alpha<<<nb, kBlock, 0, st>>>(v, l);
    k_adj_density<<<nb, kBlock, 0, st>>>(v, l);
    if (d3) k_adj_out<3><<<nb, kBlock, 0, st>>>(v, l.x, l.u, gx_in, gv_in, 0);
    else k_adj_out<2><<<nb, kBlock, 0, st>>>(v, l.x, l.u, gx_in, gv_in, 0);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TSPH_OK : fail_text(TSPH_ERR_CUDA, cudaGetErrorString(e));
}

int tsph_density_adjoint(tsph_ctx *c, tsph_tape *t, int slot, const float *grho, float *gx, void *stream) {
    int rc = check_slot(c, t, slot);
    if (rc) return rc;
    if (!grho || !gx) return fail_text(TSPH_ERR_INVALID, "null gradient pointer");
    cudaStream_t st = (cudaStream_t)stream;
    rc = sync_meta(*t, st);
    if (rc) return rc;
    rc = usable(*t, slot);
    if (rc) return rc;
    const SlotView v = slot_view(*t, slot);
    const int nb = blocks_for(v.n);
    const Lam l = lam_of(*t);
    k_adj_in_density<<<nb, kBlock, 0, st>>>(v, l, grho);
    k_adj_density<<<nb, kBlock, 0, st>>>(v, l);
    if (c->k.dim == 3) k_adj_out<3><<<nb, kBlock, 0, st>>>(v, l.x, nullptr, gx, nullptr, 1);
    else k_adj_out<2><<<nb, kBlock, 0, st>>>(v, l.x, nullptr, gx, nullptr, 1);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TSPH_OK : fail_text(TSPH_ERR_CUDA, cudaGetErrorString(e));
}

}  // extern "C"
