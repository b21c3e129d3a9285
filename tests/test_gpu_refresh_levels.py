"""A refresh of an uploaded tree in two launches (all leaves, then the internal levels on one
cluster) against one launch per level, which level ranges that do not follow one
another take (here: an empty range at the end): node COMs and the state after a step are
equal bit for bit. One-node trees, single levels, many levels, leaves of more than 16
particles, massless particles."""
import numpy as np
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200 import morton_tree as mt
from galaxy_sim_b200.nbody_gpu import NBodyGPU

pytestmark = pytest.mark.gpu

KW = dict(dt=0.005, G=1.0, epsilon=0.05, theta=0.5)


@pytest.mark.parametrize("n,kind", [(1, "disk"), (17, "disk"), (1000, "disk"), (20011, "disk"), (150000, "disk"),
                                    (3000, "coincident"), (3000, "massless")])
def test_refresh_in_two_launches_equals_one_per_level(gpu_lib, n, kind):
    g = ic.galaxy_disk(n, 60) if n > 16 else ic.hernquist_sphere(n, 60)
    P0 = g.particles.copy()
    if kind == "coincident":
        P0[500:1500, :3] = P0[500, :3]
    if kind == "massless":
        P0[::3, 3] = 0.0
        P0[1000:1400, 3] = 0.0
    b = mt.sortAndBuild(P0, g.stellar, n)
    tree, P = b["tree"], b["sorted"].reshape(-1, 8)
    moved = P.copy()
    moved[:, :3] += np.float32(0.01) * P[:, 4:7]
    out = []
    for ranges in (tree.levelRanges, tree.levelRanges + [[0, 0]]):
        sim = NBodyGPU(0, P, b["sortedStellar"])
        sim.updateParams(**KW)
        sim.uploadBHTree(tree.nodes, tree.numNodes, ranges)
        sim.writeState(moved)
        sim.encodeRefresh()
        nodes, _, _ = sim.getTree(want_perm=False)
        sim.step()
        out.append((nodes.copy(), sim.readState()[0]))
        assert sim.deviceErrors() == 0
        sim.destroy()
    assert np.array_equal(out[0][0].view(np.uint8), out[1][0].view(np.uint8))
    assert np.array_equal(out[0][1].view(np.uint32), out[1][1].view(np.uint32))
