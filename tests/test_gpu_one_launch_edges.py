"""The one-launch substep where its blocks could disagree or its context be left in a
state that the next call takes for another (needs a GPU).

Each case is held to the separate kernels, or to a context that never met it, bit
for bit.
"""
import pytest

import tests.test_gpu_one_launch as one
from tests.test_gpu_grid_edges import _need_cuda

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
