"""Node COMs of the tile kernel (block-local sums, arrivals at the nodes that span tiles)
against gs_refresh on the same tree, whose kernel carries every leaf's COM to the root
over global memory: equal bit for bit, and again after a second rebuild (the arrival
counters end at zero). Sizes around the tile of 1024 particles and above the one-cluster
rebuild's limit; coincident particles (leaves and chains of nodes that span many
tiles); pools with galaxies side by side; both COM modes."""
import numpy as np
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200._lib import check, lib
from galaxy_sim_b200.nbody_gpu import NBodyGPU
from galaxy_sim_b200.pool import GalaxyPool

pytestmark = pytest.mark.gpu

KW = dict(dt=0.005, G=1.0, epsilon=0.05, theta=0.5)


def _particles(n, kind):
    g = ic.hernquist_sphere(n, 300 + n)
    P = g.particles.copy()
    if kind == "coincident":
        P[n // 4:3 * n // 4, :3] = P[n // 4, :3]
    if kind == "all":
        P[:, :3] = 0.5
    if kind == "outlier":
        P[-1, :3] = (3.0e4, -2.0e4, 1.0e4)
    return P, g.stellar


def _equal(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("com", [0, 2])
@pytest.mark.parametrize("n,kind", [(32769, "sphere"), (65537, "sphere"), (300001, "sphere"), (50000, "coincident"),
                                    (40000, "all"), (50000, "outlier")])
def test_tile_coms_equal_refresh(gpu_lib, oracle, n, kind, com):
    P, S = _particles(n, kind)
    sim = NBodyGPU(0, P, S)
    sim.updateParams(**KW)
    sim.setComMode(com)
    for _ in range(2):
        sim.sortBuild()
        built, lr, _ = sim.getTree()
        sim.encodeRefresh()
        refreshed, _, _ = sim.getTree()
        assert _equal(built, refreshed)
    want = oracle.sort_and_build(P, S)
    assert np.array_equal(lr, want["levelRanges"])
    for f in ("isLeaf", "first", "count", "children", "size"):
        assert np.array_equal(built[f], want["nodes"][f]), f
    assert sim.deviceErrors() == 0
    sim.destroy()


@pytest.mark.parametrize("com", [0, 2])
def test_tile_coms_equal_refresh_in_a_pool(gpu_lib, com):
    sizes = [1, 16, 17, 1023, 1024, 1025, 2048, 5000, 40001]
    pool = GalaxyPool(sum(-(-n // 256) * 256 for n in sizes), len(sizes))
    check(lib().gs_set_com_mode(pool._ctx, com), pool._ctx)
    kinds = ["sphere", "sphere", "all", "coincident", "sphere", "outlier", "coincident", "all", "sphere"]
    slots = [pool.add(*_particles(n, k), KW) for n, k in zip(sizes, kinds)]
    for _ in range(2):
        pool.sort_build()
        built = [pool.get_tree(s)[0].copy() for s in slots]
        pool.refresh()
        for s, b in zip(slots, built):
            assert _equal(b, pool.get_tree(s)[0])
            assert pool.device_errors(s) == 0
    pool.close()
