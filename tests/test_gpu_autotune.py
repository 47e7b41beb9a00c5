"""The threads-per-particle tuner keeps the one-launch step where there is one (needs a
GPU)."""
import pytest

from tests.test_gpu_grid_edges import _need_cuda
from tests.test_gpu_one_launch import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 5000), (3, 900)])
def test_tuned_small_scene_steps_in_one_launch(dim, n):
    _need_cuda()
    s = _solver(dim, n, 90, False, True, inside=True)
    times = s.autotune(reps=2)
    assert set(times) == {1, 2, 4, 8} and s.tpp == 1
    s.substep()
    assert s.stats()["launches_per_step"] == 1
    s.close()


def test_separate_launches_take_the_fastest_setting():
    _need_cuda()
    for use_graph, candidates in ((False, (1, 2, 4, 8)), (True, (2, 4, 8))):
        s = _solver(3, 900, 90, False, use_graph, inside=True)
        times = s.autotune(candidates=candidates, reps=2)
        assert times[s.tpp] == min(times.values())
        s.close()
