"""The velocity map's two forms give the same field (needs a GPU).

Between steps the map packs the particles into sorted records; while a step
composed call by call is under way, whose buffers the records would take, it
reads the caller's arrays per candidate.  A grid built for the composed step from
the positions the map reads holds every particle in its current cell, so both
forms see the same particles (in another order: sums of at most ~60 FP32 terms,
1e-5 of the largest node velocity).
"""
import pytest
import torch

from tests.test_gpu_grid_edges import _need_cuda
from tests.test_gpu_one_launch import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 600), (3, 33), (3, 900)])
def test_map_between_steps_and_within_one(dim, n):
    _need_cuda()
    from tichi_sph_gb300 import Grid
    s = _solver(dim, n, 50, False, True)
    s.substep()
    s.fluid.vel[:n] = torch.randn(n, dim, generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    s.neighbor_stats()  # the grid of the positions as they are now
    g = Grid(s.config, device="cuda")
    s.map_velocity(g)
    packed = g.vel.clone()
    s.grid_build()
    g.vel.fill_(7.0)
    s.map_velocity(g)
    scale = float(packed.abs().max())
    assert float((g.vel - packed).abs().max()) <= 1e-5 * max(scale, 1e-30)
    s.close()
