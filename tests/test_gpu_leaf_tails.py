"""Leaves that run past their tile of 1024 sorted particles: node COMs and leaf ranges of the
tile kernel against gs_refresh on the same tree, bit for bit, for leaves that end just past
the tile, at and around the chunks of eight loads, in a later tile, and at the galaxy's
end. Particles at the two corners of the box make the first and the last leaf."""
import numpy as np
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200._lib import check, lib
from galaxy_sim_b200.nbody_gpu import NBodyGPU
from galaxy_sim_b200.pool import GalaxyPool

pytestmark = pytest.mark.gpu

KW = dict(dt=0.005, G=1.0, epsilon=0.05, theta=0.5)


def _galaxy(n, first, last):
    g = ic.hernquist_sphere(n, 400 + n)
    P = g.particles.copy()
    lo, hi = P[:, :3].min(0), P[:, :3].max(0)
    P[:first, :3] = lo
    P[n - last:, :3] = hi
    return P, g.stellar


def _check(tree, refreshed, n, first, last):
    assert np.array_equal(tree.view(np.uint8), refreshed.view(np.uint8))
    leaves = tree[tree["isLeaf"] == 1]
    leaves = leaves[np.argsort(leaves["first"])]
    assert np.array_equal(np.cumsum(leaves["count"])[:-1], leaves["first"][1:])   # they tile the particles
    assert leaves["count"][0] >= first and leaves["count"][-1] >= last


@pytest.mark.parametrize("com", [0, 2])
@pytest.mark.parametrize("first,last", [(1024, 1024), (1025, 1031), (1032, 1033), (1040, 2047), (2048, 2049),
                                        (2055, 3000), (3072, 17), (5001, 1)])
def test_leaf_tails_equal_refresh(gpu_lib, com, first, last):
    n = 33001
    sim = NBodyGPU(0, *_galaxy(n, first, last))
    sim.updateParams(**KW)
    sim.setComMode(com)
    for _ in range(2):
        sim.sortBuild()
        built = sim.getTree()[0].copy()
        sim.encodeRefresh()
        _check(built, sim.getTree()[0], n, first, last)
    assert sim.deviceErrors() == 0
    sim.destroy()


@pytest.mark.parametrize("com", [0, 2])
def test_leaf_tails_in_a_pool(gpu_lib, com):
    cases = [(1025, 20, 1005), (3000, 1500, 1500), (2049, 2048, 1), (4096, 1031, 2056), (5000, 1024, 3976)]
    pool = GalaxyPool(sum(-(-n // 256) * 256 for n, _, _ in cases), len(cases))
    check(lib().gs_set_com_mode(pool._ctx, com), pool._ctx)
    slots = [pool.add(*_galaxy(*c), KW) for c in cases]
    pool.sort_build()
    built = [pool.get_tree(s)[0].copy() for s in slots]
    pool.refresh()
    for s, b, c in zip(slots, built, cases):
        _check(b, pool.get_tree(s)[0], *c)
        assert pool.device_errors(s) == 0
    pool.close()
