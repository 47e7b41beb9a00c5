"""The velocity map where a velocity has a component that is not finite (needs a GPU).

The map adds X / psi W v over the candidates of a node's template cells, W = 0 for
those beyond h, to each component on its own: an infinite component gives infinity
within h and NaN (0 times it) beyond, a NaN gives NaN, and neither touches the other
components.
"""
import numpy as np
import pytest
import torch

from tests.test_gpu_grid_edges import H, _need_cuda
from tests.test_gpu_one_launch import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 600), (3, 900)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("composed", [False, True])
def test_one_component_not_finite(dim, n, value, composed):
    _need_cuda()
    from tichi_sph_gb300 import Grid
    s = _solver(dim, n, 50, False, True, inside=True)
    s.substep()
    s.fluid.vel[:n] = torch.randn(n, dim, generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    s.neighbor_stats()  # the grid of the positions as they are now
    if composed:
        s.grid_build()
    g = Grid(s.config, device="cuda")
    s.map_velocity(g)
    base = g.vel.clone()
    assert bool(base.isfinite().all())
    i = n // 2
    s.fluid.vel[i, 0] = value
    g.vel.fill_(7.0)
    s.map_velocity(g)
    assert torch.equal(g.vel[..., 1:], base[..., 1:])
    x, want = g.vel[..., 0].cpu().numpy(), base[..., 0].cpu().numpy()
    off = g.pos.cpu().numpy().astype(np.float64) - s.fluid.pos[i].cpu().numpy().astype(np.float64)
    r, box = np.sqrt((off ** 2).sum(-1)) / H, np.abs(off).max(-1) / H
    within, beyond, far = r < 0.999, (r > 1.001) & (box < 0.999), box > 2.001
    assert within.any() and beyond.any()
    assert (x[within] == np.inf).all() if value == np.inf else np.isnan(x[within]).all()
    assert np.isnan(x[beyond]).all()
    assert (x[far] == want[far]).all()
    s.close()
