"""The launch tuner's default candidates are different launches: at most 7 walk blocks fit
an SM at any walk group size, so every walk grid it times differs from the others, and
a lone galaxy whose rebuild is one kernel (no sort tiles) is timed at one tile depth."""
import pytest

from galaxy_sim_b200 import autotune as at


def test_walk_grid_candidates_differ():
    assert len({min(b, 7) for b in at.WALK_BLOCKS}) == len(at.WALK_BLOCKS)


@pytest.mark.gpu
@pytest.mark.parametrize("n,depths", [(5000, 1), (40000, 3)])
def test_sort_depths_are_timed_where_there_are_tiles(gpu_lib, n, depths):
    from galaxy_sim_b200 import initial_conditions as ic
    from galaxy_sim_b200.nbody_gpu import NBodyGPU

    g = ic.galaxy_disk(n, 3)
    sim = NBodyGPU(0, g.particles, g.stellar)
    sim.updateParams(dt=0.001, G=1.0, epsilon=0.05, theta=0.5)
    res = at.autotune(sim, steps=1, warmup=1, walk_groups=(0,), walk_splits=(0,))
    assert len([k for k in res["ms"] if "x" in k]) == depths * len(at.WALK_BLOCKS)
    sim.destroy()
