// The one-launch step of small scenes (small.cuh): its rule, its launch and the 3D
// instances (small2.cu holds the 2D ones).
#include "small.cuh"

namespace tsph {

extern template cudaError_t launch_small_dim<2>(tsph_ctx &, const SmallArgs &, int, cudaStream_t);

// One-scene contexts on the default settings (the solver loops on the device, one
// thread per particle) whose options the kernel has, up to 512 warps of
// particles per SM.  What separate launches lose (about 90 us at 1M particles:
// drained and refilled SMs, tail reductions, while nodes) shrinks beside the
// work as scenes grow, and a fixed share of the particles per SM, 32 warps
// resident, is the weaker schedule for the sweeps themselves.  Separate launches
// and one launch, us per substep (fluid particles of a 3D dam break): 8k 235 / 154,
// 27k 236 / 170, 99k 352 / 250, 205k 518 / 423, 343k 721 / 606, 1M 1619 / 1533,
// 4.1M 5632 / 6185; in 2D 61k 189 / 111, 300k 406 / 274, 1M 928 / 865.
constexpr int64_t kSmallWarpsPerSm = 512;

bool small_step_fits(const tsph_ctx &c, const tsph_set &f, const tsph_set &b) {
    if (c.n_scenes != 1 || c.batch || !c.sms || !c.scan_r1 || c.tpp != 1 || f.n < 1) return false;
    if (c.p.fbm_enabled && c.k.P != 2) return false;
    return (f.n + 31) / 32 + (b.n + 31) / 32 <= kSmallWarpsPerSm * c.sms;
}

cudaError_t launch_small_step(tsph_ctx &c, const tsph_set &f, const tsph_set &b, bool with_cfl, float *density_out,
                              cudaStream_t st) {
    SmallArgs a = {};
    a.f = f;
    a.b = b;
    a.x = c.X;
    a.with_cfl = with_cfl ? 1 : 0;
    a.st_on = c.st_on;
    a.wc = c.p.wcsph_enabled;
    a.density_out = density_out;
    if (c.rec_tape) {
        a.tape = c.rec_tape->a;
        a.record = 1;
        a.slot = c.rec_slot;
    }
    const int threads = coop_threads((f.n + 31) / 32 + (b.n + 31) / 32, c.sms);
    return c.k.dim == 3 ? launch_small_dim<3>(c, a, threads, st) : launch_small_dim<2>(c, a, threads, st);
}

}  // namespace tsph
