// Neighbour sweeps of one substep, per particle: density + alpha and the neighbour
// list, the Jacobi pair of the two pressure solves, the advection forces
// (viscosity, surface tension).  The kernels of sweeps.cu run one of them over
// all particles; the one-launch step of small scenes (small.cu) runs them one
// after another.  NC: the data they read comes from an earlier launch (read-only
// loads) or may come from this one.
#pragma once

#include "ctx.h"

namespace tsph {

// ----------------------------------------------------------------------------- density
// s + e accumulates a sum with the rounding error of every addition kept in e
// (Knuth's TwoSum, exact for any order of the terms).  The density sweep sums
// the fluid's density and compression this way: psi - psi0, which the pressure
// solves start from, cancels all but ~1e-3 (DFSPH) or ~1e-6 (VFSPH) of psi, so
// an FP32 sum's own rounding (a few 1e-7 of psi over ~40 terms) would be a
// large part of it; with the error term the sum is exact to about one rounding
// of psi, and psi's low part is kept beside it (FluidBuf::psilo).
// (The two-lane instructions, add.rn.f32x2 and sub.rn.f32x2, did not keep the
// remainder here: the results were those of a plain sum.)
__device__ __forceinline__ void acc2(float &s, float &e, float y) {
    const float t = __fadd_rn(s, y);
    const float yp = __fsub_rn(t, s);
    const float sp = __fsub_rn(t, yp);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, sp), __fsub_rn(y, yp)));
    s = t;
}

// Sums of the density sweep for one fluid particle; rho_e, comp_e: the rounding
// errors of the additions to rho and comp.
struct DensAcc {
    float rho, comp, rho_e, comp_e;
    float wsum, a2, a1x, a1y, a1z, pacc;
    int zeros;  // entries at the particle's own position (r = 0)
};

// One recorded pair (0 < r < h known) of the density sweep's list pass: the
// density and alpha terms and, with P0, k_psi's pair term for the divergence
// solve's first iteration -- one distance, one reciprocal square root and one
// spline gradient serve all of them.  The gradient factor is formed in k_psi's
// order, ((W'(q) sig / h) / r) X_j, so the psi term is k_psi's bit for bit.
// FLUIDJ: the neighbour is a fluid particle (alpha_2 has no boundary term,
// main.py:194-195).  A neighbour at the particle's own position (r = 0) is counted:
// density_exact then does the particle again.
template <bool FLUIDJ, bool P0>
__device__ __forceinline__ void density_list_pair(const Geo &g, float4 pi, float4 pj, float2 mv, float4 vi,
                                                  float4 vj, DensAcc &a) {
    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    float r;
    const float ri = pair_rinv(r2, r);
    a.zeros += !(r2 > 0.f);
    const float q = r * g.inv_h;
    const float w = kw(q) * g.sig;
    a.wsum += w;
    acc2(a.rho, a.rho_e, __fmul_rn(w, mv.x));
    acc2(a.comp, a.comp_e, __fmul_rn(w, mv.y));
    const float wg = kwg(q) * g.sig_h;
    const float f = wg * ri * pj.w;
    a.a1x += f * dx;
    a.a1y += f * dy;
    a.a1z += f * dz;
    if (FLUIDJ) a.a2 += __fdividef(wg * wg * pj.w * pj.w, mv.x);
    if (P0) a.pacc += f * (dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z));
}

// Appends neighbour entries to sorted particle s's list, four at a time: a block
// is collected in registers and stored as one int4 (a store per entry, each to its
// own 16-byte piece of L2, took the density sweep 4% longer at 1M particles).
struct ListWriter {
    int4 *wp;
    int64_t stride;
    int4 blk;
    int n, cap;
    __device__ __forceinline__ ListWriter(int *list, int64_t s, int64_t stride_, int cap_)
        : wp(reinterpret_cast<int4 *>(list) + s), stride(stride_), blk(make_int4(0, 0, 0, 0)), n(0), cap(cap_) {}
    __device__ __forceinline__ void put(int j) {
        blk = make_int4(blk.y, blk.z, blk.w, j);
        ++n;
        if ((n & 3) == 0 && n <= cap) {
            *wp = blk;
            wp += stride;
        }
    }
    // stores the last, partly filled block
    __device__ __forceinline__ void finish() {
        const int t = n & 3;
        if (t == 0 || n > cap) return;
        if (t == 1) blk.x = blk.w;
        else if (t == 2) { blk.x = blk.z; blk.y = blk.w; }
        else { blk.x = blk.y; blk.y = blk.z; blk.z = blk.w; }
        *wp = blk;
    }
};

// The density sums of a particle with others at its exact position, or with
// more neighbours than the first scan could record: the scan with the range tests
// per candidate, which leaves the particles at r = 0 out of the list (their W(0)
// terms go straight into the sums), then the arithmetic over the list; a list
// that overflows without them too gives the sums of one scan and the overflow
// mark.  Rare, so kept out of line.
template <int DIM, bool M, bool NC>
__device__ __noinline__ void density_exact(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc, int cur,
                                           int64_t s, bool psi0, DensAcc &out) {
    const SceneConst &c = scene<M>(k, sc);
    const SceneStep &st = k.ss[sc];
    Geo g;
    g.load(c, k.R);
    const long long f_shift = shift_of<M>(st.f_shift), b_shift = shift_of<M>(st.b_shift);
    const float4 pi = F.pos[s];
    const float4 *vin = F.vadv + cur * F.cap;
    const float4 vi = psi0 ? vin[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float w0 = kw(0.f) * g.sig;
    DensAcc a = {};
    bool ok;
    const long long code = cell_code<DIM>(pi, g, ok);
    ListWriter w(F.nbr, s, F.cap, k.nbr_max);
    int nfl = 0;
    auto scan = [&](const float4 *P, const float2 *mvs, int j) {
        const float4 pj = P[j];
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < g.h2) {
            if (r2 > 0.f) {
                w.put(j);
            } else {
                a.wsum += w0;
                const float2 mv = mvs[j];
                acc2(a.rho, a.rho_e, __fmul_rn(w0, mv.x));
                acc2(a.comp, a.comp_e, __fmul_rn(w0, mv.y));
            }
        }
    };
    if (ok) {
        visit_candidates_within<DIM, 1, NC>(F.start, g, pi, code, f_shift, 0, [&](int j) { scan(F.pos, F.mv, j); });
        nfl = w.n;
        visit_candidates_within<DIM, 1, NC>(B.start, g, pi, code, b_shift, 0, [&](int j) { scan(B.pos, B.mv, j); });
        w.finish();
    }
    if (w.n <= w.cap) {
        walk_blocks<1, kListOwn>(F.nbr, s, F.cap, 0, nfl, w.n,
            [&](int j) { density_list_pair<true, true>(g, pi, F.pos[j], F.mv[j], vi, vin[j], a); },
            [&](int j) { density_list_pair<false, true>(g, pi, B.pos[j], B.mv[j], vi, B.vadv[j], a); });
        F.nbr_cnt[s] = (unsigned int)nfl | ((unsigned int)(w.n - nfl) << 16);
    } else {
        a = {};
        auto within = [&](float4 pj) {
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            return dx * dx + dy * dy + dz * dz < g.h2;
        };
        visit_candidates<DIM, 1, NC>(F.start, g, code, f_shift, 0, [&](int j) {
            const float4 pj = F.pos[j];
            if (within(pj)) density_list_pair<true, true>(g, pi, pj, F.mv[j], vi, vin[j], a);
        });
        visit_candidates<DIM, 1, NC>(B.start, g, code, b_shift, 0, [&](int j) {
            const float4 pj = B.pos[j];
            if (within(pj)) density_list_pair<false, true>(g, pi, pj, B.mv[j], vi, B.vadv[j], a);
        });
        F.nbr_cnt[s] = kNbrOverflow;
    }
    out = a;
}

// Whether the density sweep does the divergence solve's first psi sweep.
__device__ __forceinline__ bool density_does_psi(const SceneConst &c, double compression) {
    return c.f_n > 0 && ((0 < c.iter_min) || (compression > (double)c.div_tol));
}

// The results of the density sweep of one particle from its sums; returns its share
// of the scene's psi_sum (0 without psi0).
__device__ __forceinline__ double density_store(const KConst &k, const FluidBuf &F, int sc, int cur, bool psi0,
                                                float4 pi, const DensAcc &a, int64_t s) {
    const float4 mp = F.mpsi[s];
    float alpha = __fmaf_rn(a.a1z, a.a1z, __fmaf_rn(a.a1y, a.a1y, __fmul_rn(a.a1x, a.a1x))) / mp.x + a.a2;
    if (alpha < 1e-4f) alpha = 1e-4f;
    // the compensated sums rounded once; psi keeps the remainder as its low part
    const float rho_f = __fadd_rn(a.rho, a.rho_e), comp_f = __fadd_rn(a.comp, a.comp_e);
    const float psi = k.vfsph ? comp_f : rho_f;
    const float psilo = k.vfsph ? __fsub_rn(a.comp_e, __fsub_rn(comp_f, a.comp))
                                : __fsub_rn(a.rho_e, __fsub_rn(rho_f, a.rho));
    F.dens[s] = make_float4(a.wsum, rho_f, comp_f, a.a2);
    F.a1[s] = make_float4(a.a1x, a.a1y, a.a1z, alpha);  // w: alpha again, for the write-back
    F.psilo[s] = psilo;
    F.mpsi[s] = make_float4(mp.x, psi, mp.z, alpha);
    // psi also rides in the current v_adv's unused w (the velocity sweeps carry
    // it along), so the advection sweep gets it with the neighbour's v_adv
    F.vadv[(int64_t)cur * F.cap + s].w = psi;
    if (psi0) {
        // IPPE_adv_psi_init + IPPE_psi_adv_non_negative, as k_psi
        float pa = ((psi - mp.z) + psilo) + a.pacc * k.sp[sc].dt;
        if (pa < 0.f) pa = 0.f;
        const float kap = pa / alpha;
        F.psiadv[s] = pa;
        F.kappa[s] = kap;
        F.pk[s] = make_float4(pi.x, pi.y, pi.z, kap);
        return (double)(pa / mp.z);
    }
    return 0.0;
}

// SPH_clean_value + SPH_prepare_attr (f,f)(f,b) + SPH_prepare_alpha_1 (f,f)(f,b)
// + SPH_prepare_alpha_2 (f,f) + SPH_prepare_alpha (sph.py:22-38, 50-105), and the
// neighbour list of the step.
//
// Two phases keep the warps converged: the candidate scan only tests r < h and
// records the pairs, then the recorded list is walked for the kernel
// arithmetic.  Bound by instruction issue and, nearly as much, by L1 wavefronts
// (216k particles: 260 warp instructions per particle, L1 at 68%): the scan tests
// without a branch (visit_hits_r1), and what only a few particles need is out of
// line (density_exact).  64 registers, 4 blocks per SM: at 80 or 48 registers 1M
// particles take 391 and 395 us against 365 (48 registers spill the scan's
// loads in flight); scan and arithmetic as two launches took 389 us.  From
// 463 us before (one test and branch per candidate, 40 registers); 205k
// particles 120 -> 100 us, 8k 78 -> 41 us.
//
// The divergence solve's first psi sweep (k_psi's work for its iteration 0) is
// done here as well when that solve will run
// (iter_min > 0 or the carried-over compression above the tolerance, the test
// k_solve_begin makes): its pair terms need only positions and the v_adv the
// solve starts from, both fixed here, and walk the same pairs in the same
// order as k_psi with one thread per particle, with the same arithmetic; the
// scene's psi_sum goes through the same partials and ticket.  psi_ready tells
// k_psi to skip that iteration (64 batched scenes: 1,794 -> 1,739 us a substep).
//
// Returns the particle's share of the scene's psi_sum (0 without psi0).
template <int DIM, bool M, bool R1, bool NC>
__device__ __forceinline__ double density_fluid_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                                     const SceneConst &c, const SceneStep &st, int cur, bool psi0,
                                                     int64_t s) {
    Geo g;
    g.load(c, k.R);
    const float4 pi = F.pos[s];
    const float4 *vin = F.vadv + cur * F.cap;
    bool ok;
    const long long code = cell_code<DIM>(pi, g, ok);
    // phase 1: every particle within h but s itself, in candidate order, fluid
    // first (particles at its exact position are still among them)
    ListWriter w(F.nbr, s, F.cap, k.nbr_max);
    int nfl = 0;
    if (ok) {
        const int self = (int)s;
        auto ff = [&](int j) {
            if (j != self) w.put(j);
        };
        auto fb = [&](int j) { w.put(j); };
        if (R1) {
            visit_hits_r1<DIM, NC>(F.start, F.pos, g, pi, code, shift_of<M>(st.f_shift), ff);
            nfl = w.n;
            if (!rows_empty_r1<DIM, NC>(B.start, g, code))
                visit_hits_r1<DIM, NC>(B.start, B.pos, g, pi, code, shift_of<M>(st.b_shift), fb);
        } else {
            auto within = [&](const float4 *P, int j) {
                const float4 pj = ld_ro<NC>(P + j);
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                return dx * dx + dy * dy + dz * dz < g.h2;
            };
            visit_candidates_within<DIM, 1, NC>(F.start, g, pi, code, shift_of<M>(st.f_shift), 0, [&](int j) {
                if (within(F.pos, j)) ff(j);
            });
            nfl = w.n;
            visit_candidates_within<DIM, 1, NC>(B.start, g, pi, code, shift_of<M>(st.b_shift), 0, [&](int j) {
                if (within(B.pos, j)) fb(j);
            });
        }
        w.finish();
    }
    const bool fits = w.n <= w.cap;
    F.nbr_cnt[s] = fits ? ((unsigned int)nfl | ((unsigned int)(w.n - nfl) << 16)) : kNbrOverflow;
    // phase 2: the arithmetic over the recorded pairs
    DensAcc a = {};
    if (fits) {
        // a particle in the grid is its own candidate, at r = 0
        if (s - c.f_slot < st.f_in) {
            const float w0 = kw(0.f) * g.sig;
            a.wsum = w0;
            const float2 mv = F.mv[s];
            acc2(a.rho, a.rho_e, __fmul_rn(w0, mv.x));
            acc2(a.comp, a.comp_e, __fmul_rn(w0, mv.y));
        }
        if (psi0) {
            const float4 vi = vin[s];
            walk_blocks<1, kListOwn>(F.nbr, s, F.cap, 0, nfl, w.n,
                [&](int j) { density_list_pair<true, true>(g, pi, F.pos[j], F.mv[j], vi, vin[j], a); },
                [&](int j) { density_list_pair<false, true>(g, pi, B.pos[j], B.mv[j], vi, B.vadv[j], a); });
        } else {
            walk_blocks<1, kListOwn>(F.nbr, s, F.cap, 0, nfl, w.n,
                [&](int j) { density_list_pair<true, false>(g, pi, F.pos[j], F.mv[j], pi, pi, a); },
                [&](int j) { density_list_pair<false, false>(g, pi, B.pos[j], B.mv[j], pi, pi, a); });
        }
    }
    if (!fits || a.zeros) {
        DensAcc e;  // (a itself stays in registers)
        density_exact<DIM, M, NC>(k, F, B, sc, cur, s, psi0, e);
        a = e;
    }
    return density_store(k, F, sc, cur, psi0, pi, a, s);
}

// The boundary's own sums: SPH_prepare_attr (b,b)(b,f), SPH_prepare_alpha_2 (b,f),
// SPH_prepare_alpha (sph.py:50-105 as called by main.py:190-197).
template <int DIM, bool M, bool R1, bool NC>
__device__ __forceinline__ void density_bound_item(const KConst &k, const FluidBuf &F, const BoundBuf &B,
                                                   const SceneConst &c, const SceneStep &st, const ScenePersist &sp,
                                                   int64_t s) {
    // the (b,b) terms of the last sweep still hold when the gather found every
    // boundary position and mass unchanged (a static boundary)
    const bool cached = sp.bb_valid && !st.b_dirty && sp.bb_n == c.b_n;
    Geo g;
    g.load(c, k.R);
    const float4 pi = B.pos[s];
    bool ok;
    const long long code = cell_code<DIM>(pi, g, ok);
    float wsum = 0.f, rho = 0.f, comp = 0.f, a2 = 0.f;
    if (ok) {
        if (cached) {
            const float4 bb = B.bb[s];
            wsum = bb.x;
            rho = bb.y;
            comp = bb.z;
        } else {
            // (B.pos is not written here: the read-only path, as in the fluid sweep)
            auto bb_pair = [&](int j) {
                const float4 pj = ld_ro<NC>(&B.pos[j]);
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 < g.h2) {
                    const float2 mv = B.mv[j];
                    float r;
                    pair_rinv(r2, r);
                    const float w = kw(r * g.inv_h) * g.sig;
                    wsum += w;
                    rho += w * mv.x;
                    comp += w * mv.y;
                }
            };
            if (R1) visit_hits_r1<DIM, NC>(B.start, B.pos, g, pi, code, shift_of<M>(st.b_shift), bb_pair);
            else visit_candidates_within<DIM, 1, NC>(B.start, g, pi, code, shift_of<M>(st.b_shift), 0, bb_pair);
            B.bb[s] = make_float4(wsum, rho, comp, 0.f);
        }
        auto bf_pair = [&](int j) {
            const float4 pj = ld_ro<NC>(&F.pos[j]);
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < g.h2) {
                const float2 mv = F.mv[j];
                float r;
                const float ri = pair_rinv(r2, r);
                const float q = r * g.inv_h;
                const float w = kw(q) * g.sig;
                wsum += w;
                rho += w * mv.x;
                comp += w * mv.y;
                if (r2 > 0.f) {
                    const float wg = kwg(q) * g.sig_h;
                    a2 += __fdividef(wg * wg * pj.w * pj.w, mv.x);
                }
            }
        };
        if (R1) {
            if (!rows_empty_r1<DIM, NC>(F.start, g, code))
                visit_hits_r1<DIM, NC>(F.start, F.pos, g, pi, code, shift_of<M>(st.f_shift), bf_pair);
        } else visit_candidates_within<DIM, 1, NC>(F.start, g, pi, code, shift_of<M>(st.f_shift), 0, bf_pair);
    }
    const float m = B.mv[s].x;
    float alpha = 0.f / m + a2;
    if (alpha < 1e-4f) alpha = 1e-4f;
    B.dens[s] = make_float4(wsum, rho, comp, a2);
    B.alpha[s] = alpha;
    const float kb = B.kappa[s] / alpha;  // boundary psi_adv / alpha (psi_adv is never advanced)
    B.kappa[s] = kb;
    B.pk[s] = make_float4(pi.x, pi.y, pi.z, kb);
}

// ----------------------------------------------------------------------------- solver
// IPPE_adv_psi_init + IPPE_psi_adv_non_negative of one particle from its pair sum;
// returns its share of the scene's psi_sum.
__device__ __forceinline__ double psi_store(const FluidBuf &F, float4 pi, float4 mp, float psilo, float dt, float acc,
                                            int64_t s) {
    float psi = ((mp.y - mp.z) + psilo) + acc * dt;
    if (psi < 0.f) psi = 0.f;
    const float kap = psi / mp.w;
    F.psiadv[s] = psi;
    F.kappa[s] = kap;
    F.pk[s] = make_float4(pi.x, pi.y, pi.z, kap);
    return (double)(psi / mp.z);
}

// Sweep A of one particle (the TPP lanes of ln): psi_adv and kappa; returns its
// share of the scene's psi_sum (in the particle's first lane).
template <int DIM, int TPP, bool M, bool NC>
__device__ __forceinline__ double psi_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                           const SceneConst &c, const SceneStep &st, int cur, const Lanes<TPP> &ln,
                                           int64_t s, bool act) {
    Geo g;
    g.load(c, k.R);
    const float4 *vin = F.vadv + cur * F.cap;
    float acc = 0.f;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = pi;
    if (act) {
        pi = F.pos[s];
        vi = vin[s];
        // IPPE_adv_psi pair term; list entries load both neighbour arrays at once
        auto term = [&](const float4 *P, const float4 *V, int j, auto listed) {
            constexpr bool L = decltype(listed)::value;
            const float4 pj = P[j];
            float4 vj = make_float4(0.f, 0.f, 0.f, 0.f);
            if (L) vj = V[j];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (L || (r2 < g.h2 && r2 > 0.f)) {
                if (!L) vj = V[j];
                float r;
                const float ri = pair_rinv(r2, r);
                const float f = kwg(r * g.inv_h) * g.sig_h * ri * pj.w;
                acc += f * (dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z));
            }
        };
        // branchy list walk: two float4 gathers per entry leave no registers
        // for a whole block's gathers at six blocks per SM
        for_each_neighbor_tpp<DIM, true, TPP, M, NC>(c, st, k.R, F, B, s, ln.q, pi,
            [&](int j, auto listed) { term(F.pos, vin, j, listed); },
            [&](int j, auto listed) { term(B.pos, B.vadv, j, listed); });
    }
    acc = ln.sum(acc);
    return act && ln.q == 0 ? psi_store(F, pi, F.mpsi[s], F.psilo[s], k.sp[sc].dt, acc, s) : 0.0;
}

// m: mass, vi: the current v_adv.
__device__ __forceinline__ void vel_store(const FluidBuf &F, int cur, float4 pi, float ki, float4 a1, float m,
                                          float4 vi, float dt, float sx, float sy, float sz, int64_t s) {
    const float Xi = pi.w;
    // (written out: wherever it is inlined, the same products are fused)
    const float ax = __fmaf_rn(Xi, sx, __fmul_rn(ki, a1.x)), ay = __fmaf_rn(Xi, sy, __fmul_rn(ki, a1.y)),
                az = __fmaf_rn(Xi, sz, __fmul_rn(ki, a1.z));
    float4 *vout = F.vadv + (1 - cur) * F.cap;
    const float sc_ = -(1.f / dt) / m;
    vout[s] = make_float4(vi.x + sc_ * ax, vi.y + sc_ * ay, vi.z + sc_ * az, vi.w);  // w: psi
}

// Sweep B of one particle (the TPP lanes of ln), into the other v_adv buffer.
template <int DIM, int TPP, bool M, bool NC>
__device__ __forceinline__ void vel_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                         const SceneConst &c, const SceneStep &st, int cur, const Lanes<TPP> &ln,
                                         int64_t s, bool act) {
    Geo g;
    g.load(c, k.R);
    // IPPE_update_vel_adv's pair term (kappa_i X_j + kappa_j X_i) g x_ij, g =
    // W'(r) / r, summed as kappa_i alpha_1,i + X_i sum_j kappa_j g x_ij:
    // alpha_1 = sum_j X_j g x_ij over the same pairs is the density sweep's,
    // and the second sum needs of a neighbour only (x, y, z, kappa), one
    // float4 written by the psi sweep (the boundary's by its density sweep)
    float sx = 0.f, sy = 0.f, sz = 0.f;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) {
        pi = F.pos[s];
        // (valid = false: a padding call of a list block, computed and dropped)
        auto term = [&](const float4 *PK, int j, auto listed, bool valid) {
            constexpr bool L = decltype(listed)::value;
            const float4 qj = PK[j];
            const float dx = pi.x - qj.x, dy = pi.y - qj.y, dz = pi.z - qj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (L || (r2 < g.h2 && r2 > 0.f)) {
                float r;
                const float ri = pair_rinv(r2, r);
                const float f = qj.w * (kwg(r * g.inv_h) * g.sig_h * ri);
                sx = valid ? sx + f * dx : sx;
                sy = valid ? sy + f * dy : sy;
                sz = valid ? sz + f * dz : sz;
            }
        };
        for_each_neighbor_tpp<DIM, true, TPP, M, NC>(c, st, k.R, F, B, s, ln.q, pi,
            [&](int j, auto listed, bool v) { term(F.pk, j, listed, v); },
            [&](int j, auto listed, bool v) { term(B.pk, j, listed, v); });
    }
    sx = ln.sum(sx);
    sy = ln.sum(sy);
    sz = ln.sum(sz);
    if (act && ln.q == 0)
        vel_store(F, cur, pi, F.kappa[s], F.a1[s], F.mpsi[s].x, F.vadv[cur * F.cap + s], k.sp[sc].dt, sx, sy, sz, s);
}

// ----------------------------------------------------------------------------- advection
__device__ __forceinline__ void normal_store(const FluidBuf &F, const Geo &g, float nx, float ny, float nz,
                                             int64_t s) {
    // w: what the surface-tension pass reads of a neighbour beside its normal
    const float w = F.vf[s] > 0.99f ? F.mpsi[s].y : __uint_as_float(kNoSurfTension);
    F.normal[s] = make_float4(nx * g.h, ny * g.h, nz * g.h, w);
}

// First pass of SPH_advection_surface_tension_acc, sph.py:134-150: surface normals.
template <int DIM, int TPP, bool M, bool NC>
__device__ __forceinline__ void normal_item(const KConst &k, const FluidBuf &F, const BoundBuf &B,
                                            const SceneConst &c, const SceneStep &st, const Lanes<TPP> &ln, int64_t s,
                                            bool act) {
    Geo g;
    g.load(c, k.R);
    float nx = 0.f, ny = 0.f, nz = 0.f;
    if (act) {
        const float4 pi = F.pos[s];
        for_each_neighbor_tpp<DIM, false, TPP, M, NC>(c, st, k.R, F, B, s, ln.q, pi,
            [&](int j, auto listed) {
                constexpr bool L = decltype(listed)::value;
                const float4 pj = F.pos[j];
                float psij = 0.f;
                if (L) psij = F.mpsi[j].y;
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (L || (r2 < g.h2 && r2 > 0.f)) {
                    if (!L) psij = F.mpsi[j].y;
                    float r;
                    const float ri = pair_rinv(r2, r);
                    const float f = -__fdividef(pj.w, psij) * (kwg(r * g.inv_h) * g.sig_h) * ri;
                    nx += f * dx;
                    ny += f * dy;
                    nz += f * dz;
                }
            },
            [&](int, auto) {});
    }
    nx = ln.sum(nx);
    ny = ln.sum(ny);
    nz = ln.sum(nz);
    if (act && ln.q == 0) normal_store(F, g, nx, ny, nz, s);
}

template <int DIM>
__device__ __forceinline__ void advect_store(const KConst &k, const FluidBuf &F, int sc, const SceneConst &c, int cur,
                                             float4 vi, float vx, float vy, float vz, float sx, float sy, float sz,
                                             float gs, float vs, int64_t s) {
    float4 *vout = F.vadv + (1 - cur) * F.cap;
    const float dt = k.sp[sc].dt;
    const float mu = (c.mu * vs) / F.rho0[s];
    const float ax = c.g[0] * gs + vx * mu + sx;
    const float ay = c.g[1] * gs + vy * mu + sy;
    const float az = (DIM == 3 ? c.g[2] * gs : 0.f) + vz * mu + sz;
    F.acc[s] = make_float4(ax, ay, az, 0.f);
    F.vel[s] = vi;
    vout[s] = make_float4(vi.x + ax * dt, vi.y + ay * dt, vi.z + az * dt, 0.f);
}

// SPH_vel_adv_2_vel + SPH_advection_gravity_acc + SPH_advection_viscosity_acc
// + (pass 2 of) SPH_advection_surface_tension_acc + SPH_advection_update_vel_adv,
// sph.py:108-166, 247-262.  The list gives the pairs within h: viscosity and,
// for a particle with surface tension (phase-0 volume fraction above 0.99), the
// cohesion term of every such neighbour (zero beyond h).  The curvature term
// has no kernel weight, so -- like the reference -- it runs over every
// candidate of the template cells, not only those within h: a second loop over
// the cells that reads each candidate's normal and psi in one load.  Its only
// distance test, r > 0, needs no position: the terms it would drop are exactly
// zero, the particle's own (n_i - n_i) and that of a particle at its exact
// position (the two have the same neighbours in the same order, each leaving
// the other out, so the same normal bit for bit).  A particle whose list overflowed takes the
// reference's form with the range tests per candidate.  gs / vs scale the
// gravity / viscosity terms by 1 or 0 (kernel-level calls may leave either
// out; x * 1 is exact, so the full step's bits are unchanged).
template <int DIM, bool ST, int TPP, bool M, bool NC>
__device__ __forceinline__ void advect_item(const KConst &k, const FluidBuf &F, const BoundBuf &B, int sc,
                                            const SceneConst &c, const SceneStep &st, int cur, const Lanes<TPP> &ln,
                                            int64_t s, bool act, float gs, float vs) {
    Geo g;
    g.load(c, k.R);
    const float4 *vin = F.vadv + cur * F.cap;
    float vx = 0.f, vy = 0.f, vz = 0.f;   // viscosity sum
    float sx = 0.f, sy = 0.f, sz = 0.f;   // surface tension sum
    float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) {
        const float4 pi = F.pos[s];
        vi = vin[s];
        const float4 mpi = F.mpsi[s];
        const float4 ni = ST ? F.normal[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        const bool st_i = ST && has_surf_tension(ni);
        const float lap = 2.f * (2.f + DIM);
        const float eps = 0.01f * g.h2;
        const float gamma = c.gamma, c_coh = c.c_coh;
        const long long f_shift = shift_of<M>(st.f_shift);
        // every term of one candidate, with the reference's range tests
        auto pair = [&](int j) {
            const float4 pj = F.pos[j];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (!(r2 > 0.f)) return;
            const bool near = r2 < g.h2;
            float r = 0.f, ri = 0.f, mj = 0.f;
            if (near) {
                const float4 vj = vin[j];
                const float4 mpj = F.mpsi[j];
                mj = mpj.x;
                ri = pair_rinv(r2, r);
                const float wg = kwg(r * g.inv_h) * g.sig_h;
                const float adx = (vi.x - vj.x) * dx + (vi.y - vj.y) * dy + (vi.z - vj.z) * dz;
                const float f = __fdividef(lap * __fdividef(pj.w, mpj.y) * wg * ri * adx, eps + r2);
                vx += f * dx;
                vy += f * dy;
                vz += f * dz;
            }
            if (ST && st_i) {
                const float4 nj = F.normal[j];   // w: the neighbour's psi
                if (has_surf_tension(nj)) {
                    const float coh = near ? -gamma * mj * (kcoh(r * g.inv_h) * c_coh) * ri : 0.f;
                    const float fac = __fdividef(2.f * mpi.z, mpi.y + nj.w);
                    sx += fac * (coh * dx + gamma * (ni.x - nj.x));
                    sy += fac * (coh * dy + gamma * (ni.y - nj.y));
                    sz += fac * (coh * dz + gamma * (ni.z - nj.z));
                }
            }
        };
        const bool exact = ST && st_i && F.nbr_cnt[s] == kNbrOverflow;
        bool ok = false;
        long long code = 0;
        if (ST && st_i) code = cell_code<DIM>(pi, g, ok);
        if (exact) {
            if (ok) visit_candidates<DIM, TPP, NC>(F.start, g, code, f_shift, ln.q, pair);
        } else {
            // list entries skip the range tests and load their neighbour's v_adv
            // and psi together with its position
            for_each_neighbor_tpp<DIM, false, TPP, M, NC>(c, st, k.R, F, B, s, ln.q, pi,
                [&](int j, auto listed) {
                    constexpr bool L = decltype(listed)::value;
                    if (!L) {
                        pair(j);  // (a particle with surface tension is not here)
                        return;
                    }
                    const float4 pj = F.pos[j];
                    const float4 vj = vin[j];
                    const float psij = vj.w;  // the neighbour's psi, set by the density sweep
                    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    float r;
                    const float ri = pair_rinv(r2, r);
                    const float wg = kwg(r * g.inv_h) * g.sig_h;
                    const float adx = (vi.x - vj.x) * dx + (vi.y - vj.y) * dy + (vi.z - vj.z) * dz;
                    // the two quotients by __fdividef (within 2 ulp, far inside the
                    // 1e-5 bar), as on every per-pair path of these sweeps
                    const float f = __fdividef(lap * __fdividef(pj.w, psij) * wg * ri * adx, eps + r2);
                    vx += f * dx;
                    vy += f * dy;
                    vz += f * dz;
                    if (ST && st_i) {
                        const float4 nj = F.normal[j];
                        if (has_surf_tension(nj)) {
                            const float mj = F.mv[j].x;
                            const float coh = -gamma * mj * (kcoh(r * g.inv_h) * c_coh) * ri;
                            const float fac = __fdividef(2.f * mpi.z, mpi.y + nj.w);
                            sx += fac * (coh * dx);
                            sy += fac * (coh * dy);
                            sz += fac * (coh * dz);
                        }
                    }
                },
                [&](int, auto) {});
            if (ST && st_i && ok) {
                // the curvature term over every candidate of the template cells
                visit_candidates<DIM, TPP, NC>(F.start, g, code, f_shift, ln.q, [&](int j) {
                    const float4 nj = F.normal[j];
                    if (has_surf_tension(nj)) {
                        const float fac = __fdividef(2.f * mpi.z, mpi.y + nj.w);
                        sx += fac * (gamma * (ni.x - nj.x));
                        sy += fac * (gamma * (ni.y - nj.y));
                        sz += fac * (gamma * (ni.z - nj.z));
                    }
                });
            }
        }
    }
    vx = ln.sum(vx);
    vy = ln.sum(vy);
    vz = ln.sum(vz);
    if (ST) {
        sx = ln.sum(sx);
        sy = ln.sum(sy);
        sz = ln.sum(sz);
    }
    if (act && ln.q == 0) advect_store<DIM>(k, F, sc, c, cur, vi, vx, vy, vz, sx, sy, sz, gs, vs, s);
}

}  // namespace tsph
