"""The one-launch substep where its blocks could disagree or its context be left in a
state that the next call takes for another (needs a GPU).

Each case is held to the separate kernels, or to a context that never met it, bit
for bit.
"""
import ctypes as C
import functools

import pytest
import torch

import tests.test_gpu_one_launch as one
from tests.test_gpu_grid_edges import H, _need_cuda
from tichi_sph_gb300 import _native

pytestmark = pytest.mark.gpu


def _solver(monkeypatch, config, *args, **kw):
    """test_gpu_one_launch's solver with other entries in its configuration."""
    scene = one._scene

    def with_config(dim, cells):
        cfg, scen, span = scene(dim, cells)
        cfg.update(config)
        return cfg, scen, span

    with monkeypatch.context() as m:
        m.setattr(one, "_scene", with_config)
        return one._solver(*args, **kw)


def _same_scalars(xs, ys):
    for x, y in zip(xs, ys):
        for k in one.SCALARS:
            assert x[k] == y[k] or (x[k] != x[k] and y[k] != y[k]), k


@pytest.mark.parametrize("dim,n,nb", [(2, 700, 90), (3, 900, 300), (3, 5000, 0), (3, 25000, 400)])
def test_no_iteration_floor(monkeypatch, dim, n, nb):
    """Without a floor of iterations the divergence solve's first test reads the
    compression carried over, above the tolerance here, which the solve replaces by
    one below it: one iteration, whether the last block holds particles (the last
    two sizes) or not."""
    _need_cuda()
    runs = []
    for use_graph in (True, False):
        s = _solver(monkeypatch, {"solver_iter_threshold_min": 0, "solver_divergence_threshold": 1e6,
                                  "solver_compression_threshold": 1e6}, dim, n, nb, False, use_graph, inside=True)
        stats = []
        for _ in range(200):
            s.set_state(0.0, 0.0, 1e7)
            s.substep()
            stats.append(s.stats())
        assert {(x["div_iter"], x["incom_iter"]) for x in stats} == {(1, 0)}
        runs.append((s, stats))
    (a, sa), (b, sb) = runs
    _same_scalars(sa, sb)
    one._same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("dim,n,nb", [(2, 700, 90), (3, 900, 300), (3, 45000, 0)])
def test_given_up_step(dim, n, nb):
    """A step whose first grid barrier waits in vain (for a block that there is not)
    leaves the particles' state and clean counters: the step enqueued behind it is
    the one that it would have been, and the next reading of the scalars fails, once."""
    _need_cuda()
    runs = []
    for fault in (True, False):
        s = one._solver(dim, n, nb, False, True, inside=n > 5000)
        s.substep()
        assert s.stats()["launches_per_step"] == 1
        if fault:
            _native.check(s._lib.tsph_set_absent_blocks(s.ctx, 1), "absent")
            s.substep()
            _native.check(s._lib.tsph_set_absent_blocks(s.ctx, 0), "absent")
        s.substep()
        if fault:
            with pytest.raises(RuntimeError, match="gave up"):
                s.stats()
        stats = [s.stats()]
        s.substep()
        stats.append(s.stats())
        runs.append((s, stats))
    (a, sa), (b, sb) = runs
    _same_scalars(sa, sb)
    one._same(a, b)
    a.close()
    b.close()


def test_recording_of_a_given_up_step():
    """The recording of a step that gave up, and of one behind it, is refused; after
    the failure has been read a new recording is not."""
    _need_cuda()
    s = one._solver(3, 900, 300, False, True, inside=True)
    tape = C.c_void_p()
    _native.check(s._lib.tsph_tape_create(s.ctx, 2, 110, C.byref(tape)), "tape")
    f, b = s._sets()
    g = torch.zeros(900, 3, device="cuda")
    gmu = torch.zeros(1, dtype=torch.float64, device="cuda")
    ptr = lambda t, c=C.c_float: C.cast(t.data_ptr(), C.POINTER(c))  # noqa: E731

    def record(absent):
        _native.check(s._lib.tsph_set_absent_blocks(s.ctx, absent), "absent")
        _native.check(s._lib.tsph_substep_record(s.ctx, f, b, tape, 1 - absent, None), "record")

    def reverse(slot):
        rc = s._lib.tsph_substep_adjoint(s.ctx, tape, slot, ptr(g), ptr(g), ptr(g), ptr(g), ptr(gmu, C.c_double), None)
        torch.cuda.synchronize()
        return rc

    start = s.fluid.pos.clone(), s.fluid.vel.clone()
    record(1)
    record(0)
    assert reverse(0) == reverse(1) == _native.ERR_STATE
    with pytest.raises(RuntimeError, match="gave up"):
        s.stats()
    s.fluid.pos.copy_(start[0])
    s.fluid.vel.copy_(start[1])
    record(0)
    assert reverse(1) == _native.OK
    s._lib.tsph_tape_destroy(tape)
    s.close()


@pytest.mark.parametrize("dim,n", [(2, 700), (3, 25000), (3, 45000)])
def test_given_up_reverse(dim, n):
    """A reverse whose grid barrier waits in vain gives gradients that are all NaN and
    a failure at the next reading of the scalars; the next reverse is not touched."""
    _need_cuda()
    s = one._solver(dim, n, 90, False, True, inside=True)
    tape = C.c_void_p()
    _native.check(s._lib.tsph_tape_create(s.ctx, 1, 110, C.byref(tape)), "tape")
    f, b = s._sets()
    _native.check(s._lib.tsph_substep_record(s.ctx, f, b, tape, 0, None), "record")
    s.stats()
    out = []
    for absent in (0, 1, 0):
        gen = torch.Generator("cuda").manual_seed(1)
        gx, gv = (torch.randn(n, dim, generator=gen, device="cuda") for _ in range(2))
        gmu = torch.zeros(1, dtype=torch.float64, device="cuda")
        ptr = lambda t, c=C.c_float: C.cast(t.data_ptr(), C.POINTER(c))  # noqa: E731
        _native.check(s._lib.tsph_set_absent_blocks(s.ctx, absent), "absent")
        _native.check(s._lib.tsph_substep_adjoint(s.ctx, tape, 0, ptr(gx), ptr(gv), ptr(gx), ptr(gv),
                                                  ptr(gmu, C.c_double), None), "reverse")
        if absent:
            with pytest.raises(RuntimeError, match="gave up"):
                s.stats()
            assert all(bool(t.isnan().all()) for t in (gx, gv, gmu))
        else:
            s.stats()
            out.append((gx, gv, gmu))
    for x, y in zip(*out):
        assert bool(x.isfinite().all()) and torch.equal(x, y)
    s._lib.tsph_tape_destroy(tape)
    s.close()


def test_replay_of_a_density_captured_with_host_loops():
    """A density evaluation captured while the solver loops run on the host: its
    replays leave counts behind, also for the one-launch steps of later."""
    _need_cuda()
    n, runs = 900, []
    for captured in (True, False):
        s = one._solver(3, n, 300, False, False, inside=True)
        tape = C.c_void_p()
        _native.check(s._lib.tsph_tape_create(s.ctx, 1, 110, C.byref(tape)), "tape")
        rho = torch.zeros(n, device="cuda")
        s.substep()

        def density():
            f, b = s._sets()
            _native.check(s._lib.tsph_density_record(s.ctx, f, b, tape, 0, C.cast(rho.data_ptr(), C.POINTER(C.c_float)),
                                                     s._stream()), "density")

        density()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                density()
        s.set_graph_mode(True)
        for _ in range(3):
            s.substep()
            graph.replay() if captured else density()
        s.substep()
        assert s.stats()["launches_per_step"] == 1
        runs.append((s, rho, tape))
    one._same(runs[0][0], runs[1][0])
    assert torch.equal(runs[0][1], runs[1][1])
    for s, _, tape in runs:
        s._lib.tsph_tape_destroy(tape)
        s.close()


def test_scalars_after_the_rest_of_a_composed_step():
    """Phase calls that go on after a whole step change the scalars on the device: a
    reading gives those, not what the step left in host memory."""
    _need_cuda()
    runs = []
    for use_graph in (True, False):
        s = one._solver(3, 900, 300, False, use_graph, inside=True)
        s.grid_build()
        s.density_alpha()
        s.substep()
        s.update()
        runs.append((s, [s.stats()]))
    assert runs[0][1][0]["steps"] == 2
    _same_scalars(runs[0][1], runs[1][1])
    for s, _ in runs:
        s.close()


@pytest.mark.parametrize("dim,cells,n", [(2, 1500, 700), (2, 1700, 700), (3, 130, 900), (3, 143, 900)])
def test_few_particles_in_a_large_grid(monkeypatch, dim, cells, n):
    """Grids below and above the size from which on a block takes all its threads (2.5M
    cells with 152 SMs)."""
    _need_cuda()
    scene = one._scene

    def wide(d, c):
        cfg, scen, span = scene(d, c)
        scen["sim_env"]["sim_space_rt"] = [cells * H] * d
        return cfg, scen, span

    monkeypatch.setattr(one, "_scene", wide)
    runs = []
    for use_graph in (True, False):
        s = one._solver(dim, n, 90, False, use_graph)
        stats = []
        for _ in range(3):
            s.substep()
            stats.append(s.stats())
        assert (stats[-1]["launches_per_step"] == 1) == use_graph
        runs.append((s, stats))
    _same_scalars(runs[0][1], runs[1][1])
    one._same(runs[0][0], runs[1][0])
    for s, _ in runs:
        s.close()


@pytest.mark.parametrize("dim,n,nb", [(2, 700, 90), (3, 5000, 700), (3, 25000, 400), (3, 45000, 90), (3, 160000, 700)])
@pytest.mark.parametrize("block", ["weakly compressible", "surface tension"])
def test_optional_blocks(monkeypatch, dim, n, nb, block):
    """The weakly compressible block, and surface tension of one phase, with eight,
    four and one lanes per particle and with runs from a queue."""
    _need_cuda()
    import tichi_sph_gb300
    wc = block == "weakly compressible"
    monkeypatch.setattr(tichi_sph_gb300, "Solver", functools.partial(tichi_sph_gb300.Solver, wcsph=wc))
    runs = []
    for use_graph in (True, False):
        s = one._solver(dim, n, nb, False, use_graph, gamma=0.0 if wc else 0.07, inside=True)
        stats = []
        for _ in range(2):
            s.substep()
            stats.append(s.stats())
        assert (stats[-1]["launches_per_step"] == 1) == use_graph
        runs.append((s, stats))
    _same_scalars(runs[0][1], runs[1][1])
    one._same(runs[0][0], runs[1][0])
    for f in ("pressure", "normal"):
        x, y = (getattr(s.fluid, f) for s, _ in runs)
        assert torch.equal(torch.nan_to_num(x.double()), torch.nan_to_num(y.double())), f
        assert bool(x.abs().max() > 0) == ((f == "pressure") == wc)
    for s, _ in runs:
        s.close()
