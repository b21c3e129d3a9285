"""Uploads are ordered with the kernels that read them: a tree of a few MB uploaded into
fresh contexts from pageable memory is complete when its conversion runs (a copy on
another stream once left its tail behind, and the tree was flagged as malformed)."""
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200 import morton_tree as mt
from galaxy_sim_b200.nbody_gpu import NBodyGPU

pytestmark = pytest.mark.gpu


def test_tree_uploads_are_complete(gpu_lib):
    n = 150000
    g = ic.galaxy_disk(n, 60)
    b = mt.sortAndBuild(g.particles, g.stellar, n)
    for _ in range(20):
        sim = NBodyGPU(0, b["sorted"], b["sortedStellar"])
        sim.uploadBHTree(b["tree"].nodes, b["tree"].numNodes, b["tree"].levelRanges)
        assert sim.deviceErrors() == 0
        sim.destroy()
