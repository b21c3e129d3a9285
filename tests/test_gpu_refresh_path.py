"""Which kernels a refresh of an uploaded tree takes: two launches where the level ranges
follow one another, one per level that has nodes where they do not, one for trees built
on the device, none for a tree without level ranges."""
import numpy as np
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200 import morton_tree as mt
from galaxy_sim_b200.nbody_gpu import NBodyGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 17, 20011])
def test_refresh_launches(gpu_lib, n):
    g = ic.hernquist_sphere(n, 60)
    b = mt.sortAndBuild(g.particles, g.stellar, n)
    tree, P = b["tree"], b["sorted"].reshape(-1, 8)
    sim = NBodyGPU(0, P, b["sortedStellar"])
    sim.updateParams(dt=0.005, G=1.0, epsilon=0.05, theta=0.5)
    assert sim.refreshKernels() == 0
    levels = tree.levelRanges
    com = []
    for ranges, kernels in ((levels, 2), (levels + [[0, 0]], len(levels)), (None, 0)):
        sim.uploadBHTree(tree.nodes, tree.numNodes, ranges)
        sim.encodeRefresh()
        assert sim.refreshKernels() == kernels
        com.append(sim.getTree(want_perm=False)[0].copy())
    assert np.array_equal(com[0].view(np.uint8), com[1].view(np.uint8))
    sim.sortBuild()
    sim.encodeRefresh()
    assert sim.refreshKernels() == 1
    assert sim.deviceErrors() == 0
    sim.destroy()
