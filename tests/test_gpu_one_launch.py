"""The one-launch substep against the separate kernels, bit for bit (needs a GPU).

With the solver loops on the device, one-scene contexts up to a size run a substep as
one cooperative kernel; with host-driven loops the same particle code runs as
separate kernels.  Both add every sum in the same order, so after three
substeps every field and every scalar must be equal -- at sizes around the
warp and the 256-slot block, with capacities beyond the particle count,
particles outside the grid, and no boundary.
"""
import numpy as np
import pytest
import torch

from tests.test_gpu_grid_edges import H, _cloud, _need_cuda, _scene

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "vel_adv", "acce_adv", "alpha_1", "mass", "rest_density", "volume_frac", "W", "sph_density",
          "sph_compression", "psi_adv", "alpha", "alpha_2", "flag", "neighb_cell_seq", "neighb_in_cell_seq",
          "neighb_cell_structured_seq")
SCALARS = ("dt", "time_count", "compression", "kinetic_energy", "potential_energy", "div_iter", "incom_iter",
           "fbm_passes", "general_flag", "status", "fluid_in_grid", "bound_in_grid", "steps", "total_div_iter",
           "total_incom_iter", "total_fbm_passes", "max_dens_compression")


def _solver(dim, n, nb, two, use_graph, gamma=0.0, inside=False):
    from tichi_sph_gb300 import Fluid, Solver, sph_config
    cfg_d, scen, span = _scene(dim, 6)
    scen["sim_env"]["gravity"] = [0.0, -9.81, 0.0][:dim]
    if gamma:
        cfg_d["solver_surface_tension_gamma"] = gamma
    if inside:  # room for the lists: about 3 (2D) or 4 (3D) particles a cell
        span = [3 * H + H * (n / (3 if dim == 2 else 4)) ** (1.0 / dim)] * dim
        scen["sim_env"]["sim_space_rt"] = span
    if two:
        cfg_d.update(solver_type="VFSPH", solver_surface_tension_gamma=0.07, solver_fbm_convection_term=50.0)
        scen["sim_env"].update(phase_num=2, phase_rest_density=[1000, 500],
                               phase_color_hex=["0x6F7DBC", "0xFA8012"])
    cfg = sph_config.Config(cfg_d, scen)
    rng = np.random.default_rng(31 * n + nb)
    sets = []
    for uid, m in enumerate((n, nb)):
        o = Fluid(m + 300, cfg, uid, device="cuda")
        o.part_num[None] = m
        pos = _cloud(rng, m, dim, span)
        if inside:  # off cell 0 too, which is no valid cell
            pos = np.clip(pos, 0.25 * H, np.asarray(span, np.float32) - 0.25 * H) + np.float32(0.0)
            pos[:, 0] = np.maximum(pos[:, 0], np.float32(1.25 * H))
        o.pos[:m] = torch.as_tensor(pos, device="cuda")
        if uid == 0:
            o.vel[:m] = torch.as_tensor(rng.normal(0, 0.3, (m, dim)).astype(np.float32), device="cuda")
        vf = rng.uniform(0, 1, m).astype(np.float32) if two else np.ones(m, np.float32)
        vf[::2] = 1.0
        vf = np.stack([vf, 1 - vf], 1) if two else vf[:, None]
        o.volume_frac[:m] = torch.as_tensor(vf, device="cuda")
        o.rest_volume[:m] = float(cfg.part_size[dim])
        o.update_mass_all()
        sets.append(o)
    return Solver(cfg, sets[0], sets[1], fbm=two, use_graph=use_graph)


@pytest.mark.parametrize("dim,n,nb,two", [(2, 1, 0, False), (2, 33, 40, False), (2, 257, 0, True),
                                          (2, 700, 90, True), (3, 31, 1, False), (3, 256, 257, False),
                                          (3, 900, 300, True), (3, 5000, 700, False), (2, 21000, 500, True),
                                          (3, 25000, 900, False), (2, 60000, 0, False),
                                          (3, 156000, 700, False), (3, 467000, 300, True)])
def test_one_launch_equals_separate_kernels(dim, n, nb, two):
    # (above 19,456 particles four lanes of a warp share one, above 38,912 one has it;
    # in 3D warps take runs from a queue above 155,648, of dealt groups from 466,944 on)
    _need_cuda()
    runs = []
    for use_graph in (True, False):
        s = _solver(dim, n, nb, two, use_graph, inside=n > 5000)
        stats = []
        for _ in range(3):
            s.substep()
            stats.append(s.stats())
        assert (stats[-1]["launches_per_step"] == 1) == use_graph
        runs.append((s, stats))
    (a, sa), (b, sb) = runs
    for x, y in zip(sa, sb):
        for k in SCALARS:
            assert x[k] == y[k] or (x[k] != x[k] and y[k] != y[k]), k
    for oa, ob in ((a.fluid, b.fluid), (a.bound, b.bound)):
        for f in FIELDS:
            x, y = getattr(oa, f), getattr(ob, f)
            assert torch.equal(torch.nan_to_num(x.double()), torch.nan_to_num(y.double())), f
    a.close()
    b.close()


@pytest.mark.parametrize("dim,n,nb,gamma", [(2, 1, 0, 0.0), (2, 700, 90, 0.0), (3, 33, 5, 0.0), (3, 900, 300, 0.07),
                                            (3, 25000, 400, 0.0), (3, 45000, 0, 0.0)])
def test_recorded_substep_and_its_reverse(dim, n, nb, gamma):
    """Recorded in one launch, reversed in one (with eight, four or one lanes per
    particle as the size has it), against separate kernels.  The forward is
    bitwise the same; the reverse adds a particle's up to 64 pair terms in
    another order, within 64 x 2^-24 = 4e-6 of the terms' size a sweep: 1e-4 of
    the largest gradient over the seven or more sweeps."""
    _need_cuda()
    import ctypes as C

    from tichi_sph_gb300 import _native
    outs = []
    for use_graph in (True, False):
        s = _solver(dim, n, nb, False, use_graph, gamma=gamma, inside=True)
        tape = C.c_void_p()
        _native.check(s._lib.tsph_tape_create(s.ctx, 2, 110, C.byref(tape)), "tape")
        f, b = s._sets()
        gmu = torch.zeros(1, dtype=torch.float64, device="cuda")
        gen = torch.Generator("cuda").manual_seed(1)
        gx = torch.randn(n, dim, generator=gen, device="cuda")
        gv = torch.randn(n, dim, generator=gen, device="cuda") * 1e-3
        for slot in range(2):
            _native.check(s._lib.tsph_substep_record(s.ctx, f, b, tape, slot, None), "record")
        ptr = lambda t, c=C.c_float: C.cast(t.data_ptr(), C.POINTER(c))  # noqa: E731
        torch.cuda.synchronize()
        rc = s._lib.tsph_substep_adjoint(s.ctx, tape, 0, ptr(gx), ptr(gv), ptr(gx), ptr(gv), ptr(gmu, C.c_double),
                                         None)
        torch.cuda.synchronize()
        outs.append((rc, s.fluid.pos.clone(), gx, gv, gmu))
        s._lib.tsph_tape_destroy(tape)
        s.close()
    (rc0, p0, *g0), (rc1, p1, *g1) = outs
    assert rc0 == rc1 == 0, _native.lib().tsph_last_error()
    assert torch.equal(p0, p1)
    for x, y in zip(g0, g1):
        assert float((x - y).abs().max()) <= 1e-4 * max(float(y.abs().max()), 1e-30)


def _same(a, b):
    for oa, ob in ((a.fluid, b.fluid), (a.bound, b.bound)):
        for f in FIELDS:
            x, y = getattr(oa, f), getattr(ob, f)
            assert torch.equal(torch.nan_to_num(x.double()), torch.nan_to_num(y.double())), f


def test_after_a_step_of_another_size():
    """A step too large for one launch leaves other counters behind, also when its
    graph is a cached one: the one-launch steps between such steps are those of
    separate kernels, bit for bit."""
    _need_cuda()
    from tichi_sph_gb300 import Fluid, Solver, sph_config
    side, few = 137, 90   # 137^3 boundary particles: too many for one launch
    cfg_d, scen, _ = _scene(3, 6)
    scen["sim_env"]["sim_space_rt"] = [(side + 3) * H] * 3
    rng = np.random.default_rng(5)
    ax = (np.arange(side) + 1.4) * H
    lattice = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    cloud = rng.uniform(2 * H, 12 * H, (700, 3)).astype(np.float32)
    runs = []
    for use_graph in (True, False):
        cfg = sph_config.Config(cfg_d, scen)
        sets = []
        for uid, pos in enumerate((cloud, lattice)):
            o = Fluid(len(pos), cfg, uid, device="cuda")
            o.part_num[None] = len(pos)
            o.pos[:] = torch.as_tensor(pos, device="cuda")
            o.volume_frac[:] = 1.0
            o.rest_volume[:] = float(cfg.part_size[3])
            o.update_mass_all()
            sets.append(o)
        s = Solver(cfg, sets[0], sets[1], use_graph=use_graph)
        launches = []
        for n in (few, len(lattice), few, len(lattice), few):
            sets[1].part_num[None] = n
            s.substep()
            launches.append(s.stats()["launches_per_step"])
        if use_graph:
            assert [x == 1 for x in launches] == [True, False, True, False, True]
        runs.append(s)
    _same(*runs)
    for s in runs:
        s.close()


def test_after_a_replay_of_captured_calls():
    """Phase calls in a caller's graph change the context's counters and scalars at
    each replay: the steps and scalars that follow are those of direct calls."""
    _need_cuda()
    from tichi_sph_gb300 import _native

    def phases(s):
        s.grid_build()
        s.density_alpha()
        for kind in (_native.SOLVE_DIV, _native.SOLVE_DENS):
            for _ in range(2):
                s.adv_psi(kind, read=False)
                s.update_vel_adv(kind)
            if kind == _native.SOLVE_DIV:
                s.nonpressure()
        s.update()

    runs, scalars = [], []
    for captured in (True, False):
        s = _solver(3, 900, 300, False, True)
        s.substep()
        got = [s.stats()]
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                phases(s)
        for _ in range(2):
            s.substep()
            if captured:
                graph.replay()
            else:
                phases(s)
            got.append(s.stats())
            s.substep()
            got.append(s.stats())
        runs.append(s)
        scalars.append(got)
    for x, y in zip(*scalars):
        for k in SCALARS:
            assert x[k] == y[k] or (x[k] != x[k] and y[k] != y[k]), k
    _same(*runs)
    for s in runs:
        s.close()


def test_two_scenes_on_two_streams():
    """One-launch steps of two contexts, enqueued on two streams without waiting for
    one another, are those of each context alone."""
    _need_cuda()
    runs = []
    for streams in ([torch.cuda.Stream(), torch.cuda.Stream()], [torch.cuda.current_stream()] * 2):
        ss = [_solver(3, 900, 300, False, True), _solver(2, 700, 90, True, True)]
        torch.cuda.synchronize()
        for _ in range(20):
            for s, q in zip(ss, streams):
                with torch.cuda.stream(q):
                    s.substep()
        torch.cuda.synchronize()
        runs.append(ss)
    for a, b in zip(*runs):
        _same(a, b)
        a.close()
        b.close()
