"""A change of the time step between volume-fraction passes called one at a time
(needs a GPU).

A pass's fluxes are proportional to the time step (the drift velocities, made in the
first pass, keep the old one), so with it doubled before the second pass every
particle's increments are twice those of the second pass without, bit for bit: those
of particles with no neighbour flagged in the first pass too.
"""
import pytest
import torch

from tests.test_gpu_grid_edges import _need_cuda
from tests.test_gpu_one_launch import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 700), (3, 900)])
def test_doubled_before_the_second_pass(dim, n):
    _need_cuda()
    from tichi_sph_gb300 import _native
    tmp = []
    for factor in (1.0, 2.0):
        s = _solver(dim, n, 90, True, True, inside=True)
        s.cfl_condition()
        s.grid_build()
        s.density_alpha()
        s.solve(_native.SOLVE_DIV)
        s.nonpressure()
        s.solve(_native.SOLVE_DENS)
        assert s.fbm_pass() == 1
        st = s.stats()
        s.set_state(st["time_count"], factor * st["dt"], st["compression"])
        s.fbm_pass()
        s.update()
        tmp.append(s.fluid.volume_frac_tmp[:n].clone())
        s.close()
    assert bool(tmp[0].isfinite().all()) and float(tmp[0].abs().max()) > 0
    assert torch.equal(tmp[1], 2 * tmp[0])
