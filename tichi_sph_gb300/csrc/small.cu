// The one-launch step of small scenes (small.cuh): its rules and its launch.  The
// small_*d_*.cu files hold the kernel's instances.
#include "small.cuh"

namespace tsph {

#define TSPH_SMALL(D, L, Q) \
    extern template cudaError_t launch_small_lanes<D, L, Q>(tsph_ctx &, const SmallArgs &, int, cudaStream_t);
TSPH_SMALL(2, 1, false) TSPH_SMALL(2, 4, false) TSPH_SMALL(2, 8, false)
TSPH_SMALL(3, 1, true) TSPH_SMALL(3, 1, false) TSPH_SMALL(3, 4, false) TSPH_SMALL(3, 8, false)
#undef TSPH_SMALL

// One-scene contexts on the default settings (the solver loops on the device, one
// thread per particle) whose options the kernel has, up to 512 warps of
// particles per SM (fluid and boundary together).  What separate launches lose
// (drained and refilled SMs, tail reductions, while nodes) shrinks beside the work
// as scenes grow, while one launch has 32 warps resident per SM and a share of the
// particles for each SM.  Separate launches and one launch, us per substep (fluid
// particles of a 3D dam break): after 500 substeps 216k 515 / 442, 439k 795 / 716,
// 512k 893 / 809, 1M 1464 / 1385, 2.1M (past the line) 2596 / 2550, 4.1M
// 4546 / 4668; from rest 1.3k 196 / 79, 8k 211 / 93, 27k 222 / 128, 99k 318 / 226, 205k
// 487 / 409, 1M 1571 / 1497, 2.1M 2943 / 2936, 4.1M 5530 / 5631; in 2D 5k 171 / 81, 61k
// 192 / 112, 300k after 1,500 substeps 491 / 363, 900k 1430 / 1371.
constexpr int64_t kSmallWarpsPerSm = 512;
// Cells per SM from which on a block takes all its threads (launch_small_step).
constexpr int64_t kCellsPerSm = 16384;

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
    a.host_st = c.host_ss;
    a.host_sp = c.host_sp;
    a.with_cfl = with_cfl ? 1 : 0;
    a.st_on = c.st_on;
    a.wc = c.p.wcsph_enabled;
    a.density_out = density_out;
    a.absent = c.absent;
    if (c.rec_tape) {
        a.tape = c.rec_tape->a;
        a.record = 1;
        a.slot = c.rec_slot;
    }
    // lanes per particle: as many as the block's 32 warps leave for its runs of 32
    // (us a substep with one lane and with eight or four: 1.3k particles in 3D 166 /
    // 93, 8k 155 / 95, 27k 177 / 143; in 2D, a third of the neighbours, 5k 132 / 122)
    const int64_t runs = ((f.n + kBlock - 1) / kBlock * (kBlock / 32) + c.sms - 1) / c.sms;
    const int lanes = runs * 8 <= 32 ? 8 : runs * 4 <= 32 ? 4 : 1;
    // The boundary's runs have warps of their own beside them, unless one or two more
    // would take a block past 512 threads: the next size, 1,024, is slower (5k in 2D
    // 90 and 92 us for a substep and the copies of its start state) and takes all of
    // an SM's registers, so that no other context's step fits beside it (four
    // contexts of 5k on four streams, a substep each: 151 us with 512 threads, 287
    // with 1,024, 212 in separate launches; of 8k 186, 344 and 298).
    const int64_t lwarps = runs * lanes;
    int64_t bruns = ((b.n + 31) / 32 + c.sms - 1) / c.sms;
    if (lwarps <= 16 && lwarps + bruns > 16 && bruns <= 2) bruns = 16 - lwarps;
    // Few particles in a large grid: the time is that of counting its cells, which all
    // the threads that an SM holds share (us a substep with the particles' 256 or
    // 512 threads, with 1,024 and in separate launches: 2k particles in 1M cells 91 / 92
    // / 200, 4.1M 134 / 120 / 267, 64M 1637 / 1070 / 1243; 62k in 2D, 1M 110 / 111 / 183,
    // 64M 1652 / 1083 / 1224).
    const bool many_cells = c.k.total_nodes > kCellsPerSm * c.sms;
    const int threads = many_cells ? 1024 : coop_threads((lwarps + bruns) * c.sms, c.sms);
    // the kernel leaves zero counters behind, other grid builds do not
    if (!c.counts_zero) {
        cudaError_t e = cudaMemsetAsync(c.F.count, 0, sizeof(int) * c.k.total_nodes, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(c.B.count, 0, sizeof(int) * c.k.total_nodes, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(c.X.bar + kBarTailF, 0, 4 * (kBarWords - kBarTailF), st);
        if (e != cudaSuccess) return e;
    }
    // several runs a warp in 3D: taken from a queue (us a substep of a developed flow
    // with fixed turns and with the queue: 216k 478 / 442, 439k 756 / 706, 1M
    // 1614 / 1385; 205k from rest 425 / 424).  In 2D, with less work a run, it gave
    // nothing: 300k 363 / 362, 900k 1371 / 1395.
    const bool d3 = c.k.dim == 3;
    switch (lanes) {
        case 8:
            return d3 ? launch_small_lanes<3, 8, false>(c, a, threads, st)
                      : launch_small_lanes<2, 8, false>(c, a, threads, st);
        case 4:
            return d3 ? launch_small_lanes<3, 4, false>(c, a, threads, st)
                      : launch_small_lanes<2, 4, false>(c, a, threads, st);
        default:
            if (!d3) return launch_small_lanes<2, 1, false>(c, a, threads, st);
            return runs > 32 ? launch_small_lanes<3, 1, true>(c, a, threads, st)
                             : launch_small_lanes<3, 1, false>(c, a, threads, st);
    }
}

}  // namespace tsph
