// One-launch substep of a small scene: every phase of the step inside one
// cooperative kernel, grid-wide barriers between them.
//
// A scene of a few thousand particles fills a fraction of the GPU, and its
// substep as separate launches is a chain of about thirty kernels of 2 to 10 us
// (plus the while nodes of the solver loops): launch gaps, tail reductions and
// cold starts, not work.  Here a phase costs its own latency and one barrier
// (1.25 us with one block per SM and no block late), and the solver loops' tests are made by
// every block from the same sums.  The per-particle arithmetic and the order of
// every sum are those of the separate kernels, so the results are the same bit
// for bit (sweeps.cuh, grid.cuh, fbm.cuh, tape.cuh hold the particle code).
//
// Which scenes take it: see small_step_fits.
#pragma once

#include "coop.cuh"
#include "fbm.cuh"
#include "grid.cuh"
#include "lanes.cuh"
#include "sweeps.cuh"
#include "tape.cuh"
#include "wcsph.cuh"

namespace tsph {

// Kernel arguments beside the context's own structures.
struct SmallArgs {
    tsph_set f, b;
    SmallScratch x;
    SceneStep *host_st;  // pinned host copies of the scalars
    ScenePersist *host_sp;
    TapeArrays tape;
    float *density_out;  // not null: only the grid and the densities (in the caller's order), no step
    int slot;            // of the tape
    int record, with_cfl, st_on, wc;
    unsigned int absent;  // blocks that will not come (GridBarrier)
};

// Inclusive scan over the block; total in every thread.
__device__ __forceinline__ int small_block_scan(int v, int *sh, int &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int u = lane < warps ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= o) u += y;
        }
        sh[lane] = u;
    }
    __syncthreads();
    total = sh[31];
    return x + (w > 0 ? sh[w - 1] : 0);
}

// Sum of per-warp sums in the order the separate kernels add them: the eight warps
// of a 256-slot block one after another, block sums by lanes 32 apart, then the
// lanes' tree.  All threads of the block call; the result is in thread 0.
__device__ __forceinline__ double small_psi_sum(const double *warp_sums, int64_t slots, double *sh) {
    const int64_t nblk = slots / kBlock;
    const int lane = threadIdx.x & 31;
    double acc = 0.0;
    for (int64_t b0 = 0; b0 < nblk; b0 += kSmallSums) {
        const int m = (int)(nblk - b0 < kSmallSums ? nblk - b0 : kSmallSums);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const double *p = warp_sums + (b0 + i) * (kBlock / 32);
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kBlock / 32; ++q) s += __ldcg(p + q);
            sh[i] = s;
        }
        __syncthreads();
        if (threadIdx.x < 32)
            for (int i = lane; i < m; i += 32) acc += sh[i];
    }
    if (threadIdx.x < 32) acc = warp_sum(acc);
    return acc;
}

// P: phases of the volume-fraction update, 0 without it.  L: lanes per particle of
// the neighbour sweeps (lanes.cuh); with more than one, a block's warps hold all of
// its runs of 32 particles at a time (launch_small_step).  Q: warps take runs from a
// queue (for_items).
template <int DIM, bool ST, int P, int L, bool Q>
struct SmallStep {
    const KConst &k;
    const FluidBuf &F;
    const BoundBuf &B;
    const SmallArgs &a;
    GridBarrier bar;
    RunQueue queue;
    double *sh_d;
    int *sh_i;
    int64_t ns;  // the fluid's slots in whole blocks of the separate kernels
    int cur;  // the current v_adv buffer: the same in every thread of the grid

    __device__ __forceinline__ SceneStep &st() const { return k.ss[0]; }
    __device__ __forceinline__ bool first_block() const { return blockIdx.x == 0; }
    __device__ __forceinline__ bool last_block() const { return blockIdx.x == gridDim.x - 1; }

    // With the CFL condition on, the block's largest |v|.
    __device__ __forceinline__ void largest_speed() {
        const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
        if (a.record && tid == 0) a.tape.meta[a.slot] = TapeMeta{};
        if (!a.with_cfl) return;
        float m = 0.f;
        for (int64_t i = tid; i < a.f.n; i += nt) {
            float s = 0.f;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float v = a.f.vel[i * DIM + d];
                s += v * v;
            }
            const float vn = sqrtf(s);
            if (vn > 1e-4f) m = fmaxf(m, vn);  // NaN norms fail the test, as in the reference
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float *sh = reinterpret_cast<float *>(sh_i);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, sh[w]);
            a.x.vmax[blockIdx.x] = m;
        }
    }

    // cfl_condition from the blocks' maxima (first block; k_cfl's arithmetic).
    __device__ __forceinline__ void time_step() {
        if (!a.with_cfl || !first_block() || threadIdx.x >= 32) return;
        float vm = 0.f;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) vm = fmaxf(vm, __ldcg(a.x.vmax + i));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vm = fmaxf(vm, __shfl_xor_sync(0xffffffffu, vm, o));
        if (threadIdx.x != 0) return;
        const SceneConst &c = k.s0;
        float dt = __fdiv_rn(c.part_size, (float)c.cs);
        if (vm > 1e-4f) dt = fminf(dt, __fmul_rn(__fdiv_rn(c.part_size, vm), c.cfl));
        k.sp[0].dt = dt;
        k.sp[0].time_count += (double)dt;
    }

    // The block's cells [lo, hi) of the two grids (lo a multiple of four).
    __device__ __forceinline__ void cell_range(int64_t &lo, int64_t &hi) const {
        const int64_t per = ((k.total_nodes + gridDim.x - 1) / gridDim.x + 3) & ~(int64_t)3;
        lo = blockIdx.x * per < k.total_nodes ? blockIdx.x * per : k.total_nodes;
        hi = lo + per < k.total_nodes ? lo + per : k.total_nodes;
    }
    // Few enough cells that each block adds up the counts before its own (4,096 loads
    // for each grid at the most, 4 to 16 a thread) rather than meet at a barrier for
    // the blocks' totals.
    __device__ __forceinline__ bool few_cells() const { return k.total_nodes <= 16384; }
    __device__ __forceinline__ void count_totals() {
        int64_t lo, hi;
        cell_range(lo, hi);
        for (int g = 0; g < 2; ++g) {
            const int *count = g ? B.count : F.count;
            int s = 0, total;
            for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += __ldcg(count + i);
            small_block_scan(s, sh_i, total);
            if (threadIdx.x == 0) a.x.totals[2 * blockIdx.x + g] = total;
        }
    }
    // The cells' starts; the last block sets the step's scalars.
    __device__ __forceinline__ void scan_cells() {
        int64_t lo, hi;
        cell_range(lo, hi);
        int in[2];
        for (int g = 0; g < 2; ++g) {
            const int *count = g ? B.count : F.count;
            int *start = g ? B.start : F.start;
            int before = 0, total;
            if (few_cells()) {
                const int4 *c4 = reinterpret_cast<const int4 *>(count);
                for (int64_t i = threadIdx.x; i < lo / 4; i += blockDim.x) {
                    const int4 v = __ldcg(c4 + i);
                    before += (v.x + v.y) + (v.z + v.w);
                }
                for (int64_t i = lo / 4 * 4 + threadIdx.x; i < lo; i += blockDim.x) before += __ldcg(count + i);
            } else {
                for (int i = threadIdx.x; i < (int)blockIdx.x; i += blockDim.x) before += __ldcg(a.x.totals + 2 * i + g);
            }
            small_block_scan(before, sh_i, total);
            int run = total;  // particles in the cells before this block's
            for (int64_t i0 = lo; i0 < hi; i0 += blockDim.x) {
                const int64_t i = i0 + threadIdx.x;
                const int v = i < hi ? __ldcg(count + i) : 0;
                const int incl = small_block_scan(v, sh_i, total);
                if (i < hi) start[i] = run + incl - v;
                run += total;
            }
            in[g] = run;
            if (last_block() && threadIdx.x == 0) start[k.total_nodes] = run;
        }
        if (!last_block() || threadIdx.x != 0) return;
        SceneStep z = {};
        z.f_in = in[0];
        z.b_in = in[1];
        z.f_tail = (int)__ldcg(a.x.bar + kBarTailF);
        z.b_tail = (int)__ldcg(a.x.bar + kBarTailB);
        z.status = (int)__ldcg(a.x.bar + kBarStatus);
        st() = z;
    }
    // Zero counts for the next step (no phase reads them any more).
    __device__ __forceinline__ void clear_counts() {
        int64_t lo, hi;
        cell_range(lo, hi);
        for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) F.count[i] = B.count[i] = 0;
        if (first_block() && threadIdx.x == 0) a.x.bar[kBarTailF] = a.x.bar[kBarTailB] = a.x.bar[kBarStatus] = 0;
    }

    // The warp's share of the scene's psi_sum.
    __device__ __forceinline__ void put_warp_sum(double v, int64_t warp) {
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) a.x.sums[warp] = v;
    }

    // f(lanes, slot) -> the particle's share of psi_sum, over the fluid's slots and,
    // with L > 1, L lanes per particle; the shares are summed per run of 32 slots
    // (in f's last act of the phase: the block synchronises).  fb over the
    // boundary's nb.
    template <bool SUM, class FN, class FB>
    __device__ __forceinline__ void lane_sweep(int64_t nb, FN &&f, FB &&fb) {
        if constexpr (L == 1) {
            for_items<Q>(queue, ns, nb, [&](int64_t s, int64_t w) {
                const double v = f(Lanes<1>(), s);
                if (SUM) put_warp_sum(v, w);
            }, fb);
        } else {
            lane_sweep_wide<SUM>(nb, f, fb);
        }
    }
    template <bool SUM, class FN, class FB>
    __device__ __forceinline__ void lane_sweep_wide(int64_t nb, FN &&f, FB &&fb) {
        const WarpShare fl(ns), bo(nb);
        const Lanes<L> ln;
        const int64_t mine = (int64_t)fl.runs * L, total = mine + bo.runs;
        for (int64_t w = threadIdx.x >> 5; w < total; w += blockDim.x >> 5) {
            if (w < mine) {
                const int64_t in = w * ln.PPW + ln.p;  // slot within the block's runs
                const double v = f(ln, (int64_t)fl.first * 32 + in);
                if (SUM && ln.q == 0) sh_d[in] = v;
            } else {
                fb(((int64_t)bo.first + w - mine) * 32 + (threadIdx.x & 31));
            }
        }
        if (!SUM) return;
        __syncthreads();
        for (int64_t r = threadIdx.x >> 5; r < (int64_t)fl.runs; r += blockDim.x >> 5)
            put_warp_sum(sh_d[r * 32 + (threadIdx.x & 31)], (int64_t)fl.first + r);
    }

    // One pressure solve (k_solve_begin, k_psi, k_vel); psi_done: the first psi sweep
    // has run.  Every block makes the loop test from the compression that the
    // last block derives while the others update velocities.  With psi_done the
    // first test has been made, and held, before the barrier behind the density
    // sweep; it is not made again here, where no barrier lies between it and the
    // last block's new value.  Without, a psi sweep and its barrier do.
    __device__ __forceinline__ bool solve(int kind, bool psi_done) {
        const SceneConst &c = k.s0;
        const double tol = kind == kSolveDiv ? (double)c.div_tol : (double)c.comp_tol;
        const int slot = a.slot;
        int it = 0;
        bool cond = psi_done || 0 < c.iter_min || *(volatile double *)&k.sp[0].compression > tol;
        while (cond) {
            if (!psi_done) {
                lane_sweep<true>(0, [&](const Lanes<L> &ln, int64_t s) {
                    if constexpr (L == 1) return psi_item<DIM, 1, false, false>(k, F, B, 0, c, st(), cur, ln, s, s < c.f_n);
                    else return psi_lanes<DIM, L>(k, F, B, c, st(), cur, ln, s, s < c.f_n);
                }, [](int64_t) {});
                if (!bar.sync()) return false;
            }
            psi_done = false;
            lane_sweep<false>(0, [&](const Lanes<L> &ln, int64_t s) {
                if (a.record && ln.q == 0) tape_iter_item(k, F, a.tape, slot, kind, it, cur, s);
                if constexpr (L == 1) vel_item<DIM, 1, false, false>(k, F, B, 0, c, st(), cur, ln, s, s < c.f_n);
                else vel_lanes<DIM, L>(k, F, B, c, st(), cur, ln, s, s < c.f_n);
                return 0.0;
            }, [](int64_t) {});
            ++it;
            const bool capped = it > c.iter_max;
            if (last_block()) {
                const double sum = small_psi_sum(a.x.sums, ns, sh_d);
                if (threadIdx.x == 0) {
                    st().psi_sum = sum;
                    k.sp[0].compression = sum / (double)c.f_n;
                    if (kind == kSolveDiv) st().div_iter = it;
                    else st().incom_iter = it;
                    if (capped) atomicOr(&st().status, kind == kSolveDiv ? TSPH_ST_DIV_ITER_CAP : TSPH_ST_DENS_ITER_CAP);
                }
            }
            if (!bar.sync()) return false;
            cur = 1 - cur;
            cond = !capped && (it < c.iter_min || *(volatile double *)&k.sp[0].compression > tol);
        }
        return true;
    }

    // The weakly compressible pressure block (k_wc_pressure, k_wc_acce).
    __device__ __forceinline__ bool weakly_compressible() {
        const SceneConst &c = k.s0;
        for_items<Q>(queue, c.f_n, c.b_n, [&](int64_t s, int64_t) { if (s < c.f_n) wc_pressure_fluid_item(F, c, s); },
                  [&](int64_t s) { if (s < c.b_n) wc_pressure_bound_item(B, a.b.pressure, s); });
        if (!bar.sync()) return false;
        for_items<Q>(queue, c.f_n, 0, [&](int64_t s, int64_t) {
            if (s < c.f_n) wc_acce_item<DIM, false, false>(k, F, B, 0, c, st(), cur, s);
        }, [](int64_t) {});
        return bar.sync();
    }

    // The volume-fraction update (k_fbm_drift, k_fbm_begin, k_fbm_pass).
    __device__ __forceinline__ bool mixture() {
        const SceneConst &c = k.s0;
        for_items<Q>(queue, c.f_n, 0, [&](int64_t s, int64_t) {
            if (s >= c.f_n) return;
            F.flagpass[s] = 0;
            fbm_drift_item<DIM, P ? P : 1>(k, F, 0, c, cur, s);
        }, [](int64_t) {});
        if (!bar.sync()) return false;
        int pass = 0;
        bool flagged;
        do {
            ++pass;
            for_items<Q>(queue, c.f_n, 0, [&](int64_t s, int64_t) {
                const bool neg = s < c.f_n && fbm_pass_item<DIM, P ? P : 1, false, false>(k, F, B, 0, c, st(), pass, s);
                if (__any_sync(0xffffffffu, neg) && (threadIdx.x & 31) == 0) atomicMax(&st().general_flag, pass);
            }, [](int64_t) {});
            if (!bar.sync()) return false;
            // (a block that is ahead may have raised it to the next pass already)
            flagged = *(volatile int32_t *)&st().general_flag >= pass;
        } while (flagged && pass < c.fbm_max_passes);
        if (first_block() && threadIdx.x == 0) {
            st().fbm_passes = pass;
            st().gflag_out = flagged ? 1 : 0;
            if (flagged) atomicOr(&st().status, TSPH_ST_FBM_PASS_CAP);
        }
        return true;
    }

    __device__ __forceinline__ bool run() {
        const SceneConst &c = k.s0;
        largest_speed();
        int *ctr = reinterpret_cast<int *>(a.x.bar);
        for_items<Q>(queue, a.f.n, a.b.n,
            [&](int64_t i, int64_t) {
                if (i < a.f.n) encode_item<DIM>(k, a.f, 0, F.count, F.slot, ctr + kBarTailF, ctr + kBarStatus, i);
            },
            [&](int64_t i) {
                if (i < a.b.n) encode_item<DIM>(k, a.b, 0, B.count, B.slot, ctr + kBarTailB, ctr + kBarStatus, i);
            });
        if (!bar.sync()) return false;
        if (!few_cells()) {
            count_totals();
            if (!bar.sync()) return false;
        }
        time_step();
        scan_cells();
        if (!bar.sync()) return false;
        for_items<Q>(queue, a.f.n, a.b.n,
            [&](int64_t i, int64_t) {
                if (i < a.f.n) scatter_item(k, 0, a.f.neighb_cell_seq, F.slot, F.start, F.perm_u, i);
            },
            [&](int64_t i) {
                if (i < a.b.n) scatter_item(k, 1, a.b.neighb_cell_seq, B.slot, B.start, B.perm_u, i);
            });
        if (!bar.sync()) return false;
        clear_counts();
        for_items<Q>(queue, a.f.n, a.b.n,
                  [&](int64_t u, int64_t) { if (u < a.f.n) gather_fluid_item<DIM>(k, a.f, F, c, st(), u); },
                  [&](int64_t u) { if (u < a.b.n) gather_bound_item<DIM>(k, a.b, B, c, 0, u); });
        if (!bar.sync()) return false;
        const bool psi0 = density_does_psi(c, *(volatile double *)&k.sp[0].compression);
        const int slot = a.slot;
        lane_sweep<true>(a.b.n,
            [&](const Lanes<L> &ln, int64_t s) {
                double v = 0.0;
                if constexpr (L == 1) {
                    if (s < c.f_n) v = density_fluid_item<DIM, false, true, false>(k, F, B, 0, c, st(), 0, psi0, s);
                } else {
                    v = density_fluid_lanes<DIM, L>(k, F, B, c, st(), 0, psi0, ln, s, s < c.f_n);
                }
                if (ln.q != 0) return v;
                if (a.record) tape_state_fluid_item(k, F, a.tape, slot, s);
                if (a.density_out && s < c.f_n) a.density_out[F.perm[s]] = F.dens[s].y;
                return v;
            },
            [&](int64_t s) {
                if (s >= c.b_n) return;
                density_bound_item<DIM, false, true, false>(k, F, B, c, st(), k.sp[0], s);
                if (a.record) tape_state_bound_item(k, B, a.tape, slot, s);
            });
        if (ST && a.record && a.tape.start) {
            const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
            for (int64_t i = tid; i < a.tape.nstart; i += (int64_t)gridDim.x * blockDim.x)
                a.tape.start[(int64_t)slot * a.tape.nstart + i] = F.start[i];
        }
        if (a.density_out) return true;
        if (!bar.sync()) return false;
        cur = 0;
        if (!solve(kSolveDiv, psi0)) return false;
        if (ST) {
            lane_sweep<false>(0, [&](const Lanes<L> &ln, int64_t s) {
                if constexpr (L == 1) normal_item<DIM, 1, false, false>(k, F, B, c, st(), ln, s, s < c.f_n);
                else normal_lanes<DIM, L>(k, F, B, c, st(), ln, s, s < c.f_n);
                return 0.0;
            }, [](int64_t) {});
            if (!bar.sync()) return false;
        }
        lane_sweep<false>(0, [&](const Lanes<L> &ln, int64_t s) {
            if constexpr (L == 1)
                advect_item<DIM, ST, 1, false, false>(k, F, B, 0, c, st(), cur, ln, s, s < c.f_n, 1.f, 1.f);
            else advect_lanes<DIM, ST, L>(k, F, B, c, st(), cur, ln, s, s < c.f_n);
            if (a.record && ln.q == 0) tape_vmid_item(k, F, a.tape, slot, s);
            return 0.0;
        }, [](int64_t) {});
        if (!bar.sync()) return false;
        cur = 1 - cur;
        if (!solve(kSolveDens, false)) return false;
        if (a.wc && !weakly_compressible()) return false;
        if (P && !mixture()) return false;
        double *en = a.x.sums;  // the solves' sums are done with
        for_items<Q>(queue, ns, a.b.n,
            [&](int64_t pid, int64_t w) {
                double ke = 0.0, pe = 0.0;
                if (pid < c.f_n)
                    update_fluid_item<DIM>(k, a.f, F, 0, c, st(), cur, B.start, P ? 1 : 0, a.st_on, pid, ke, pe);
                ke = warp_sum(ke);
                pe = warp_sum(pe);
                if ((threadIdx.x & 31) == 0) {
                    en[w] = ke;
                    en[ns / 32 + w] = pe;
                }
            },
            [&](int64_t pid) { if (pid < a.b.n) update_bound_item<DIM>(k, a.b, B, F.start, pid); });
        if (first_block() && threadIdx.x == 0) {
            st().cur = cur;
            if (a.record) tape_end_item(k, a.tape, slot);
        }
        return true;
    }

    // The last block to leave: the energies, the running totals, the barrier's reset,
    // and the scalars' copies in pinned host memory, so that a caller who reads them
    // after every substep waits for the kernel alone (two small copies behind it
    // cost a time loop about 25 us a substep).  After a step that was given up, zero
    // counts for the next one, which may be enqueued already, and marks that stay
    // until the caller has been told.
    __device__ __forceinline__ void leave(bool done) {
        if (!last_block_done(a.x.bar + kBarLeft, gridDim.x)) return;
        // (any block may have given up, whatever this one saw)
        const unsigned int given_up = __ldcg(a.x.bar + kBarGaveUp);
        double ke = 0.0, pe = 0.0;
        for (int64_t i = threadIdx.x; !a.density_out && i < ns / kBlock && threadIdx.x < kBlock; i += kBlock) {
            ke += coop_block_tree(a.x.sums + i * (kBlock / 32));
            pe += coop_block_tree(a.x.sums + ns / 32 + i * (kBlock / 32));
        }
        ke = coop_sum256(ke, sh_d);
        pe = coop_sum256(pe, sh_d);
        const bool ok = done && !given_up;
        if (!ok)
            for (int64_t i = threadIdx.x; i < k.total_nodes; i += blockDim.x) F.count[i] = B.count[i] = 0;
        if (threadIdx.x == 0) {
            if (!ok) {
                k.sp[0].gave_up = 1;
                a.x.bar[kBarTailF] = a.x.bar[kBarTailB] = a.x.bar[kBarStatus] = 0;
            } else if (!a.density_out) {
                st().kinetic_energy = ke;
                st().potential_energy = pe;
                step_totals(k.sp[0], st());
            }
            // (a recording behind a step given up starts from an unfinished state)
            if (a.record && k.sp[0].gave_up) atomicOr(&a.tape.meta[a.slot].status, TSPH_TAPE_GAVE_UP);
            a.x.bar[kBarCount] = a.x.bar[kBarGaveUp] = a.x.bar[kBarLeft] = 0;
        }
        __syncthreads();
        // the scalars, to their host copies
        const int i = threadIdx.x, ns4 = (int)(sizeof(SceneStep) / 4), np4 = (int)(sizeof(ScenePersist) / 4);
        if (i < ns4) reinterpret_cast<int *>(a.host_st)[i] = __ldcg(reinterpret_cast<const int *>(k.ss) + i);
        if (i < np4) reinterpret_cast<int *>(a.host_sp)[i] = __ldcg(reinterpret_cast<const int *>(k.sp) + i);
    }
};

// One block per SM; 64 registers let the largest block have 1,024 threads.
template <int DIM, bool ST, int P, int L, bool Q>
__global__ void __launch_bounds__(1024, 1) k_small_step(const __grid_constant__ KConst k,
                                                        const __grid_constant__ FluidBuf F,
                                                        const __grid_constant__ BoundBuf B,
                                                        const __grid_constant__ SmallArgs a) {
    __shared__ double sh_d[kSmallSums];
    __shared__ int sh_i[33];
    __shared__ unsigned int sh_next;
    if (Q) {
        if (threadIdx.x == 0) sh_next = 0;
        __syncthreads();
    }
    SmallStep<DIM, ST, P, L, Q> step{k, F, B, a, {a.x.bar, a.absent}, {&sh_next, 0u}, sh_d, sh_i, (a.f.n + kBlock - 1) / kBlock * kBlock, 0};
    const bool done = step.run();
    step.leave(done);
}

// The instances with DIM, L and Q (a translation unit each).
template <int DIM, int L, bool Q>
cudaError_t launch_small_lanes(tsph_ctx &c, const SmallArgs &a, int threads, cudaStream_t st) {
    const bool fbm = c.p.fbm_enabled != 0;
    if (c.st_on)
        return fbm ? launch_coop(k_small_step<DIM, true, 2, L, Q>, c.sms, threads, st, c.k, c.F, c.B, a)
                   : launch_coop(k_small_step<DIM, true, 0, L, Q>, c.sms, threads, st, c.k, c.F, c.B, a);
    return fbm ? launch_coop(k_small_step<DIM, false, 2, L, Q>, c.sms, threads, st, c.k, c.F, c.B, a)
               : launch_coop(k_small_step<DIM, false, 0, L, Q>, c.sms, threads, st, c.k, c.F, c.B, a);
}

}  // namespace tsph
