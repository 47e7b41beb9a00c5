// Weakly compressible pressure block and the particle-to-grid velocity map --
// the two per-step kernels the reference ships commented out in sph_step
// (main.py:238-242 and main.py:254).
//
// Weakly compressible block (after the density solve, before the volume-fraction
// update): WC_pressure_val (sph.py:169-176) per fluid particle,
// p = rho0 cs^2 / gamma ((rho / rho0)^7 - 1) clamped at 0 with rho the step's
// sph_density; WC_pressure_acce (sph.py:179-193) over the fluid and boundary
// pairs of the step's neighbour list, acce_adv_i -= (p_i / rho_i^2 + p_j /
// rho_j^2) m_j W'(r) x_ij / r; then SPH_advection_update_vel_adv
// (sph.py:247-250), which sets v_adv = vel + acce_adv dt and so replaces the
// density solve's correction -- the reference's semantics when the block is on.
// The boundary's pressure is whatever its set holds (the reference never
// writes it).
#include <cuda_runtime.h>

#include "ctx.h"
#include "wcsph.cuh"

namespace tsph {

namespace {

template <bool M>
__global__ void __launch_bounds__(kBlock) k_wc_pressure(KConst k, FluidBuf F, BoundBuf B, const float *bpress) {
    pdl_entry();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < F.cap) {
        const SceneConst &c = scene<M>(k, f_block_scene<M>(k, s - (s % kChunk)));
        if (s - c.f_slot < c.f_n) wc_pressure_fluid_item(F, c, s);
    }
    if (s < B.cap) {
        const SceneConst &c = scene<M>(k, b_block_scene<M>(k, s - (s % kChunk)));
        if (s - c.b_slot < c.b_n) wc_pressure_bound_item(B, bpress, s);
    }
}

template <int DIM, bool M>
__global__ void __launch_bounds__(kBlock) k_wc_acce(KConst k, FluidBuf F, BoundBuf B) {
    pdl_entry();
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int sc = f_block_scene<M>(k, blockIdx.x * (int64_t)kBlock);
    const SceneConst &c = scene<M>(k, sc);
    if (s - c.f_slot < c.f_n) wc_acce_item<DIM, M, true>(k, F, B, sc, c, k.ss[sc], k.ss[sc].cur, s);
}

// What the velocity map reads of a particle, in sorted order: the caller's
// current position, and velocity with X / psi.  p.w is X / psi too, or NaN where a
// component of the velocity is not finite: where it is finite the map need not
// read what lies beyond h, where W = 0, and elsewhere it does, as 0 times such a
// component is NaN.
template <int DIM>
__device__ __forceinline__ void map_record(const KConst &k, const tsph_set &U, int64_t pid, float4 &p, float4 &v) {
    const bool vf = k.vfsph != 0;
    const float X = vf ? U.rest_volume[pid] : U.mass[pid];
    const float psi = vf ? U.sph_compression[pid] : U.sph_density[pid];
    const float *x = U.pos + pid * DIM, *u = U.vel + pid * DIM;
    v = make_float4(u[0], u[1], DIM == 3 ? u[2] : 0.f, X / psi);
    const bool fin = isfinite(v.x) && isfinite(v.y) && isfinite(v.z);
    p = make_float4(x[0], x[1], DIM == 3 ? x[2] : 0.f, fin ? v.w : __int_as_float(0x7fffffff));
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) k_map_pack(KConst k, FluidBuf F, tsph_set U) {
    const int64_t s = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (s < k.s0.f_n) map_record<DIM>(k, U, F.perm[s], F.pk[s], F.facc[s]);
}

// map_velocity over the nodes of a regular grid, one thread per node, x fastest
// (the nodes of a warp then lie along a row of cells and share candidates; out
// is in C order).  PACKED: the particles' records are in F.pk and F.facc, which
// hold nothing between steps, one 16-byte load per candidate and the velocity
// only within h; otherwise (a step composed call by call is under way) they are
// made per candidate from the caller's arrays.  Bound by the candidate loads:
// 190k nodes over 97k particles took 167 us with nine scattered loads per
// candidate and z fastest, and takes 57 us in both launches.
template <int DIM, bool PACKED>
__global__ void __launch_bounds__(kBlock) k_map_velocity(KConst k, FluidBuf F, tsph_set U, float lb0, float lb1,
                                                         float lb2, float dist, int n0, int n1, int n2,
                                                         float *out) {
    const int64_t t = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int64_t total = (int64_t)n0 * n1 * (DIM == 3 ? n2 : 1);
    if (t >= total) return;
    const SceneConst &c = k.s0;
    const int i0 = (int)(t % n0), i1 = (int)(t / n0 % n1), i2 = DIM == 3 ? (int)(t / n0 / n1) : 0;
    const int64_t I = ((int64_t)i0 * n1 + i1) * (DIM == 3 ? n2 : 1) + i2;
    const float4 gp = make_float4(lb0 + (float)i0 * dist, lb1 + (float)i1 * dist,
                                  DIM == 3 ? lb2 + (float)i2 * dist : 0.f, 0.f);
    Geo g;
    g.load(c, k.R);
    bool ok;
    const long long code = cell_code<DIM>(gp, g, ok);
    float vx = 0.f, vy = 0.f, vz = 0.f;
    if (ok) {
        visit_candidates<DIM>(F.start, g, code, 0, 0, [&](int j) {
            float4 p, v;
            if (PACKED) p = F.pk[j];
            else map_record<DIM>(k, U, F.perm[j], p, v);
            const float dx = gp.x - p.x, dy = gp.y - p.y, dz = DIM == 3 ? gp.z - p.z : 0.f;
            const float q = sqrtf(dx * dx + dy * dy + dz * dz) * g.inv_h;
            if (q >= 1.f && isfinite(p.w)) return;  // W = 0
            if (PACKED) v = F.facc[j];
            const float f = (isfinite(p.w) ? p.w : v.w) * (kw(q) * g.sig);
            vx += f * v.x;
            vy += f * v.y;
            if (DIM == 3) vz += f * v.z;
        });
    }
    out[I * DIM] = vx;
    out[I * DIM + 1] = vy;
    if (DIM == 3) out[I * DIM + 2] = vz;
}

}  // namespace

void launch_wc(tsph_ctx &c, const tsph_set &b, cudaStream_t st) {
    const int64_t n = c.F.cap > c.B.cap ? c.F.cap : c.B.cap;
    c.launches += 2;
    if (c.n_scenes > 1) {
        TSPH_LAUNCH((k_wc_pressure<true>), blocks_for(n), kBlock, st, c.k, c.F, c.B, b.pressure);
        if (c.k.dim == 3) TSPH_LAUNCH((k_wc_acce<3, true>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B);
        else TSPH_LAUNCH((k_wc_acce<2, true>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B);
    } else {
        TSPH_LAUNCH((k_wc_pressure<false>), blocks_for(n), kBlock, st, c.k, c.F, c.B, b.pressure);
        if (c.k.dim == 3) TSPH_LAUNCH((k_wc_acce<3, false>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B);
        else TSPH_LAUNCH((k_wc_acce<2, false>), blocks_for(c.F.cap), kBlock, st, c.k, c.F, c.B);
    }
}

void set_last_error_text(const char *msg);

template <int DIM>
static void launch_map(tsph_ctx &c, const tsph_set &f, const float *lb, float dist, const int32_t *shape,
                       int64_t total, float *out, cudaStream_t st) {
    const int nb = blocks_for(total), n2 = DIM == 3 ? shape[2] : 1;
    const float lb2 = DIM == 3 ? lb[2] : 0.f;
    if (c.kl_phase == 0 && c.k.s0.f_n > 0) {
        k_map_pack<DIM><<<blocks_for(c.k.s0.f_n), kBlock, 0, st>>>(c.k, c.F, f);
        k_map_velocity<DIM, true>
            <<<nb, kBlock, 0, st>>>(c.k, c.F, f, lb[0], lb[1], lb2, dist, shape[0], shape[1], n2, out);
    } else {
        k_map_velocity<DIM, false>
            <<<nb, kBlock, 0, st>>>(c.k, c.F, f, lb[0], lb[1], lb2, dist, shape[0], shape[1], n2, out);
    }
}

}  // namespace tsph

using namespace tsph;

extern "C" int tsph_map_velocity(tsph_ctx *c, const tsph_set *f, const float *lb, float dist, const int32_t *shape,
                                 float *grid_vel, void *stream) {
    if (!c || !f || !lb || !shape || !grid_vel) {
        set_last_error_text("null argument");
        return TSPH_ERR_INVALID;
    }
    if (c->n_scenes != 1) {
        set_last_error_text("tsph_map_velocity takes a one-scene context");
        return TSPH_ERR_INVALID;
    }
    if (!c->stepped) {
        set_last_error_text("tsph_map_velocity needs the cell grid of a step");
        return TSPH_ERR_STATE;
    }
    const int dim = c->k.dim;
    int64_t total = 1;
    for (int d = 0; d < dim; ++d) {
        if (shape[d] < 1) {
            set_last_error_text("grid shape must be positive");
            return TSPH_ERR_INVALID;
        }
        total *= shape[d];
    }
    if (total > 0x7fffffffll) {
        set_last_error_text("grid too large");
        return TSPH_ERR_INVALID;
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (dim == 3) launch_map<3>(*c, *f, lb, dist, shape, total, grid_vel, st);
    else launch_map<2>(*c, *f, lb, dist, shape, total, grid_vel, st);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_error_text(cudaGetErrorString(e));
        return TSPH_ERR_CUDA;
    }
    return TSPH_OK;
}
