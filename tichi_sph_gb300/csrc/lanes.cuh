// The sweeps of one substep with L lanes per particle, for the one-launch step of
// scenes too small to fill the SMs with one thread per particle: there a sweep is
// a chain of list blocks, each a round trip to L2 for its gathers, and lanes that
// take blocks of the same particle make it one or two.
//
// The results are those of one thread per particle bit for bit: every lane
// evaluates its entries' terms, and all lanes of the particle then add the terms
// of all of them in list order (exchanged by shuffles), which replicates the
// serial sum.  The expressions are those of sweeps.cuh.  (The
// volume-fraction pass keeps one thread per particle: its sum was not the same
// in this form.)
#pragma once

#include "sweeps.cuh"

namespace tsph {

template <int N>
struct Term {
    float v[N];
};

// add(term, fluid) for the entries [0, ntot) of the particle's list in order, in
// every lane of it; term = lf(j) for the nfl fluid neighbours, lb(j) for the
// boundary's, evaluated by one lane, E at a time.  All lanes of the warp call
// (ntot = 0 without a particle).
template <int L, int E, int N, class LF, class LB, class AF>
__device__ __forceinline__ void walk_in_order(const int *nbr, int64_t s, int64_t cap, const Lanes<L> &ln, int nfl,
                                              int ntot, LF &&lf, LB &&lb, AF &&add) {
    static_assert(E == 2 || E == 4, "entries per lane and round");
    const int most = __reduce_max_sync(0xffffffffu, ntot);  // of the warp's particles
    for (int t0 = 0; t0 < most; t0 += L * E) {
        Term<N> term[E];
        const int t = t0 + ln.q * E;
        int j[E];
#pragma unroll
        for (int e = 0; e < E; ++e) j[e] = 0;
        if (t < ntot) {
            const int *p = nbr + nbr_index(t, s, cap);
            if (E == 4) {
                const int4 b = *reinterpret_cast<const int4 *>(p);
                j[0] = b.x, j[1] = b.y, j[E - 2] = b.z, j[E - 1] = b.w;
            } else {
                const int2 b = *reinterpret_cast<const int2 *>(p);
                j[0] = b.x, j[1] = b.y;
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
#pragma unroll
            for (int n = 0; n < N; ++n) term[e].v[n] = 0.f;
            if (t + e < nfl) term[e] = lf(j[e]);
            else if (t + e < ntot) term[e] = lb(j[e]);
        }
#pragma unroll 1
        for (int g = 0; g < L && t0 + g * E < most; ++g) {
            const int from = g * ln.PPW + ln.p;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                Term<N> x;
#pragma unroll
                for (int n = 0; n < N; ++n) x.v[n] = __shfl_sync(0xffffffffu, term[e].v[n], from);
                const int u = t0 + g * E + e;
                if (u < ntot) add(x, u < nfl);
            }
        }
    }
}

// Sums of one value over a particle's lanes / its first lane's value.
template <int L>
__device__ __forceinline__ int lanes_sum(const Lanes<L> &ln, int v) {
#pragma unroll
    for (int o = ln.PPW; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Whether some particle of the warp has no list (its sweeps scan the cells): the
// warp then works with one lane per particle.
__device__ __forceinline__ bool warp_has_overflow(unsigned int pc) {
    return __any_sync(0xffffffffu, pc == kNbrOverflow) != 0;
}

// ----------------------------------------------------------------------------- density
// density_fluid_item: a lane scans every L-th template row of the two grids (one
// mask per row), the hits' places in the list follow from a scan over the lanes.
template <int DIM, int L>
__device__ __forceinline__ double density_fluid_lanes(const KConst &k, const FluidBuf &F, const BoundBuf &B,
                                                      const SceneConst &c, const SceneStep &st, int cur, bool psi0,
                                                      const Lanes<L> &ln, int64_t s, bool act) {
    constexpr int RF = DIM == 3 ? 9 : 3, RT = 2 * RF, M = (RT + L - 1) / L;
    Geo g;
    g.load(c, k.R);
    const float4 pi = act ? F.pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 *vin = F.vadv + cur * F.cap;
    bool ok;
    const long long code64 = cell_code<DIM>(pi, g, ok);
    const int nx = (int)g.nx, nxny = DIM == 3 ? (int)g.nxny : 0, nn = (int)g.node_num;
    const int reach = nxny + nx + 1;
    ok = ok && act && !(code64 + reach < 1 || code64 - reach > nn - 1);
    const int code = ok ? (int)code64 : 0;
    int beg[M], num[M];
    bool longer = false;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int R = ln.q + m * L, r = R < RF ? R : R - RF;
        const int *start = R < RF ? F.start : B.start;
        const int rc = code + (r % 3 - 1) * nx + (DIM == 3 ? (r / 3 - 1) * nxny : 0);
        const int lo = max(rc - 1, 1), hi = min(rc + 1, nn - 1);
        beg[m] = num[m] = 0;
        if (ok && R < RT && lo <= hi) {
            beg[m] = start[g.cbase + lo];
            num[m] = start[g.cbase + hi + 1] - beg[m];
        }
        longer |= num[m] > 32;
    }
    // a row of more than one mask: one lane per particle
    if (__any_sync(0xffffffffu, longer))
        return act && ln.q == 0 ? density_fluid_item<DIM, false, true, false>(k, F, B, 0, c, st, cur, psi0, s) : 0.0;
    unsigned int mask[M];
    int at[M], total = 0, nf = 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int R = ln.q + m * L;
        const float4 *P = (R < RF ? F.pos : B.pos) + beg[m];
        unsigned int b = 0;
        for (int e0 = 0; e0 < num[m]; e0 += 4) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 pj = P[e0 + e];
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                b = __funnelshift_l(__float_as_uint(__fsub_rn(r2, g.h2)), b, 1);
            }
        }
        if (num[m] > 0) {
            b <<= 32 - ((num[m] + 3) & ~3);
            b &= 0xffffffffu << (32 - num[m]);
            const int self = (int)s - beg[m];
            if (R == RF / 2 && self >= 0 && self < num[m]) b &= ~(0x80000000u >> self);
        }
        mask[m] = b;
        const int n = __popc(b);
        int incl = n;
#pragma unroll
        for (int o = ln.PPW; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (ln.q * ln.PPW >= o) incl += y;
        }
        at[m] = total + incl - n;
        total += __shfl_sync(0xffffffffu, incl, (L - 1) * ln.PPW + ln.p);
        nf += R < RF ? n : 0;
    }
    const int nfl = lanes_sum(ln, nf);
    const bool fits = total <= k.nbr_max;
    if (fits) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            unsigned int b = mask[m];
            int t = at[m];
            while (b) {
                const int i = __clz(b);
                b ^= 0x80000000u >> i;
                F.nbr[nbr_index(t++, s, F.cap)] = beg[m] + i;
            }
        }
    }
    if (act && ln.q == 0) F.nbr_cnt[s] = fits ? ((unsigned int)nfl | ((unsigned int)(total - nfl) << 16)) : kNbrOverflow;
    __syncwarp();
    DensAcc a = {};
    bool zero = false;
    if (act && s < st.f_in && fits) {
        // a particle in the grid is its own candidate, at r = 0
        const float w0 = kw(0.f) * g.sig;
        a.wsum = w0;
        const float2 mv = F.mv[s];
        acc2(a.rho, a.rho_e, __fmul_rn(w0, mv.x));
        acc2(a.comp, a.comp_e, __fmul_rn(w0, mv.y));
    }
    const float4 vi = act && psi0 ? vin[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    // density_list_pair's terms
    auto term = [&](const float4 *P, const float2 *mvs, const float4 *V, int j) {
        const float4 pj = P[j];
        const float2 mv = mvs[j];
        const float4 vj = psi0 ? V[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        float r;
        const float ri = pair_rinv(r2, r);
        zero |= !(r2 > 0.f);
        const float q = r * g.inv_h;
        const float w = kw(q) * g.sig;
        const float wg = kwg(q) * g.sig_h;
        const float f = wg * ri * pj.w;
        return Term<10>{{w, __fmul_rn(w, mv.x), __fmul_rn(w, mv.y), f, dx, dy, dz,
                         dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z), wg * wg * pj.w * pj.w, mv.x}};
    };
    walk_in_order<L, 2, 10>(F.nbr, s, F.cap, ln, fits ? nfl : 0, fits ? total : 0,
        [&](int j) { return term(F.pos, F.mv, vin, j); }, [&](int j) { return term(B.pos, B.mv, B.vadv, j); },
        [&](const Term<10> &x, bool fluid) {
            a.wsum += x.v[0];
            acc2(a.rho, a.rho_e, x.v[1]);
            acc2(a.comp, a.comp_e, x.v[2]);
            a.a1x += x.v[3] * x.v[4];
            a.a1y += x.v[3] * x.v[5];
            a.a1z += x.v[3] * x.v[6];
            // (the quotient here, beside its addition: the compiler fuses the two)
            if (fluid) a.a2 += __fdividef(x.v[8], x.v[9]);
            a.pacc += x.v[3] * x.v[7];
        });
    const bool exact = lanes_sum(ln, zero ? 1 : 0) != 0 || !fits;
    if (!act || ln.q != 0) return 0.0;
    if (exact) {
        DensAcc e;
        density_exact<DIM, false, false>(k, F, B, 0, cur, s, psi0, e);
        a = e;
    }
    return density_store(k, F, 0, cur, psi0, pi, a, s);
}

// ----------------------------------------------------------------------------- solver
template <int DIM, int L>
__device__ __forceinline__ double psi_lanes(const KConst &k, const FluidBuf &F, const BoundBuf &B, const SceneConst &c,
                                            const SceneStep &st, int cur, const Lanes<L> &ln, int64_t s, bool act) {
    const unsigned int pc = act ? F.nbr_cnt[s] : 0u;
    if (warp_has_overflow(pc))
        return ln.q == 0 ? psi_item<DIM, 1, false, false>(k, F, B, 0, c, st, cur, Lanes<1>(), s, act) : 0.0;
    Geo g;
    g.load(c, k.R);
    const float4 *vin = F.vadv + cur * F.cap;
    float acc = 0.f, psilo = 0.f;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi, mp = pi;
    if (act) {
        pi = F.pos[s];
        vi = vin[s];
        mp = F.mpsi[s];  // (for the end: in flight with the rest)
        psilo = F.psilo[s];
    }
    const float dt = k.sp[0].dt;
    auto term = [&](const float4 *P, const float4 *V, int j) {
        const float4 pj = P[j], vj = V[j];
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        float r;
        const float ri = pair_rinv(r2, r);
        const float f = kwg(r * g.inv_h) * g.sig_h * ri * pj.w;
        return Term<2>{{f, dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z)}};
    };
    const int nfl = (int)(pc & 0xffffu), ntot = nfl + (int)(pc >> 16);
    walk_in_order<L, 4, 2>(F.nbr, s, F.cap, ln, nfl, ntot, [&](int j) { return term(F.pos, vin, j); },
                           [&](int j) { return term(B.pos, B.vadv, j); },
                           [&](const Term<2> &x, bool) { acc += x.v[0] * x.v[1]; });
    return act && ln.q == 0 ? psi_store(F, pi, mp, psilo, dt, acc, s) : 0.0;
}

template <int DIM, int L>
__device__ __forceinline__ void vel_lanes(const KConst &k, const FluidBuf &F, const BoundBuf &B, const SceneConst &c,
                                          const SceneStep &st, int cur, const Lanes<L> &ln, int64_t s, bool act) {
    const unsigned int pc = act ? F.nbr_cnt[s] : 0u;
    if (warp_has_overflow(pc)) {
        if (ln.q == 0) vel_item<DIM, 1, false, false>(k, F, B, 0, c, st, cur, Lanes<1>(), s, act);
        return;
    }
    Geo g;
    g.load(c, k.R);
    float sx = 0.f, sy = 0.f, sz = 0.f, ki = 0.f, m = 0.f;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), a1 = pi, vi = pi;
    if (act) {
        pi = F.pos[s];
        ki = F.kappa[s];  // (these for the end: in flight with the rest)
        a1 = F.a1[s];
        m = F.mpsi[s].x;
        vi = F.vadv[cur * F.cap + s];
    }
    const float dt = k.sp[0].dt;
    auto term = [&](const float4 *PK, int j) {
        const float4 qj = PK[j];
        const float dx = pi.x - qj.x, dy = pi.y - qj.y, dz = pi.z - qj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        float r;
        const float ri = pair_rinv(r2, r);
        return Term<4>{{qj.w * (kwg(r * g.inv_h) * g.sig_h * ri), dx, dy, dz}};
    };
    const int nfl = (int)(pc & 0xffffu), ntot = nfl + (int)(pc >> 16);
    walk_in_order<L, 4, 4>(F.nbr, s, F.cap, ln, nfl, ntot, [&](int j) { return term(F.pk, j); },
                           [&](int j) { return term(B.pk, j); },
                           [&](const Term<4> &x, bool) {
                               sx += x.v[0] * x.v[1];
                               sy += x.v[0] * x.v[2];
                               sz += x.v[0] * x.v[3];
                           });
    if (act && ln.q == 0) vel_store(F, cur, pi, ki, a1, m, vi, dt, sx, sy, sz, s);
}

// ----------------------------------------------------------------------------- advection
template <int DIM, int L>
__device__ __forceinline__ void normal_lanes(const KConst &k, const FluidBuf &F, const BoundBuf &B,
                                             const SceneConst &c, const SceneStep &st, const Lanes<L> &ln, int64_t s,
                                             bool act) {
    const unsigned int pc = act ? F.nbr_cnt[s] : 0u;
    if (warp_has_overflow(pc)) {
        if (ln.q == 0) normal_item<DIM, 1, false, false>(k, F, B, c, st, Lanes<1>(), s, act);
        return;
    }
    Geo g;
    g.load(c, k.R);
    float nx = 0.f, ny = 0.f, nz = 0.f;
    const float4 pi = act ? F.pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int nfl = (int)(pc & 0xffffu);
    walk_in_order<L, 4, 4>(F.nbr, s, F.cap, ln, nfl, nfl,
        [&](int j) {
            const float4 pj = F.pos[j];
            const float psij = F.mpsi[j].y;
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            float r;
            const float ri = pair_rinv(r2, r);
            return Term<4>{{-__fdividef(pj.w, psij) * (kwg(r * g.inv_h) * g.sig_h) * ri, dx, dy, dz}};
        },
        [](int) { return Term<4>{}; },
        [&](const Term<4> &x, bool) {
            nx += x.v[0] * x.v[1];
            ny += x.v[0] * x.v[2];
            nz += x.v[0] * x.v[3];
        });
    if (act && ln.q == 0) normal_store(F, g, nx, ny, nz, s);
}

template <int DIM, bool ST, int L>
__device__ __forceinline__ void advect_lanes(const KConst &k, const FluidBuf &F, const BoundBuf &B,
                                             const SceneConst &c, const SceneStep &st, int cur, const Lanes<L> &ln,
                                             int64_t s, bool act) {
    const unsigned int pc = act ? F.nbr_cnt[s] : 0u;
    if (warp_has_overflow(pc)) {
        if (ln.q == 0) advect_item<DIM, ST, 1, false, false>(k, F, B, 0, c, st, cur, Lanes<1>(), s, act, 1.f, 1.f);
        return;
    }
    Geo g;
    g.load(c, k.R);
    const float4 *vin = F.vadv + cur * F.cap;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 pi = act ? F.pos[s] : zero4, vi = act ? vin[s] : zero4, mpi = act ? F.mpsi[s] : zero4;
    const float4 ni = ST && act ? F.normal[s] : zero4;
    const bool st_i = ST && act && has_surf_tension(ni);
    const float lap = 2.f * (2.f + DIM), eps = 0.01f * g.h2, gamma = c.gamma, c_coh = c.c_coh;
    float vx = 0.f, vy = 0.f, vz = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
    const int nfl = (int)(pc & 0xffffu);
    constexpr int N = ST ? 6 : 4;
    walk_in_order<L, ST ? 2 : 4, N>(F.nbr, s, F.cap, ln, nfl, nfl,
        [&](int j) {
            const float4 pj = F.pos[j], vj = vin[j];
            const float psij = vj.w;
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            float r;
            const float ri = pair_rinv(r2, r);
            const float wg = kwg(r * g.inv_h) * g.sig_h;
            const float adx = (vi.x - vj.x) * dx + (vi.y - vj.y) * dy + (vi.z - vj.z) * dz;
            Term<N> t;
            t.v[0] = __fdividef(lap * __fdividef(pj.w, psij) * wg * ri * adx, eps + r2);
            t.v[1] = dx;
            t.v[2] = dy;
            t.v[3] = dz;
            if (ST) {
                t.v[N - 2] = t.v[N - 1] = 0.f;  // without surface tension: adds zeros
                if (st_i) {
                    const float4 nj = F.normal[j];
                    if (has_surf_tension(nj)) {
                        t.v[N - 2] = -gamma * F.mv[j].x * (kcoh(r * g.inv_h) * c_coh) * ri;
                        t.v[N - 1] = __fdividef(2.f * mpi.z, mpi.y + nj.w);
                    }
                }
            }
            return t;
        },
        [](int) { return Term<N>{}; },
        [&](const Term<N> &x, bool) {
            vx += x.v[0] * x.v[1];
            vy += x.v[0] * x.v[2];
            vz += x.v[0] * x.v[3];
            if (ST) {
                const float coh = x.v[N - 2], fac = x.v[N - 1];
                sx += fac * (coh * x.v[1]);
                sy += fac * (coh * x.v[2]);
                sz += fac * (coh * x.v[3]);
            }
        });
    if (ST) {
        // the curvature term over every candidate of the template cells
        bool ok = false;
        const long long code = cell_code<DIM>(pi, g, ok);
        const bool on = st_i && ok;
        constexpr int zr = DIM == 3 ? 1 : 0;
        for (int dz = -zr; dz <= zr; ++dz) {
            for (int dy = -1; dy <= 1; ++dy) {
                const long long rc = code + dy * g.nx + dz * g.nxny;
                const long long lo = rc - 1 < 1 ? 1 : rc - 1, hi = rc + 1 > g.node_num - 1 ? g.node_num - 1 : rc + 1;
                int beg = 0, end = 0;
                if (on && lo <= hi) {
                    beg = F.start[g.cbase + lo];
                    end = F.start[g.cbase + hi + 1];
                }
                for (int j0 = beg; __any_sync(0xffffffffu, j0 < end); j0 += L) {
                    const int j = j0 + ln.q;
                    float fac = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
                    if (j < end) {
                        const float4 nj = F.normal[j];
                        if (has_surf_tension(nj)) {
                            fac = __fdividef(2.f * mpi.z, mpi.y + nj.w);
                            tx = gamma * (ni.x - nj.x);
                            ty = gamma * (ni.y - nj.y);
                            tz = gamma * (ni.z - nj.z);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < L; ++q) {
                        const int from = q * ln.PPW + ln.p;
                        const float f = __shfl_sync(0xffffffffu, fac, from);
                        sx += f * __shfl_sync(0xffffffffu, tx, from);
                        sy += f * __shfl_sync(0xffffffffu, ty, from);
                        sz += f * __shfl_sync(0xffffffffu, tz, from);
                    }
                }
            }
        }
    }
    if (act && ln.q == 0)
        advect_store<DIM>(k, F, 0, c, cur, vi, vx, vy, vz, sx, sy, sz, 1.f, 1.f, s);
}

}  // namespace tsph
