"""The one-kernel rebuild of a small lone galaxy against the separate kernels, which a
pool of two galaxies runs: sorted records, permutation, tree nodes (COMs included),
level ranges, tracked centres and the state after a full step are equal bit for bit.
Sizes at the edges of blocks, threads and slices, the last size it takes and the first it
does not; coincident particles (leaves that span blocks), a far outlier (deep shared
prefixes), non-finite positions, and both COM modes."""
import numpy as np
import pytest

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200.nbody_gpu import NBodyGPU
from galaxy_sim_b200.pool import GalaxyPool

pytestmark = pytest.mark.gpu

KW = dict(dt=0.005, G=1.0, epsilon=0.05, theta=0.5, haloMass=1.0, haloA=2.0,
          haloCenters=[[0.1, 0.2, 0.3, 0.0], [1.0, 0.0, 0.0, 0.0]])


def _case(n, kind):
    g = ic.hernquist_sphere(n, 100 + n)
    P = g.particles.copy()
    if kind == "coincident":       # one leaf of half the particles, across many blocks
        P[n // 4:3 * n // 4, :3] = P[n // 4, :3]
    elif kind == "all":
        P[:, :3] = 0.5
    elif kind == "outlier":
        P[-1, :3] = (3.0e4, -2.0e4, 1.0e4)
    elif kind == "nonfinite":
        P[n // 2, 0], P[n // 3, 1] = np.nan, np.inf
    return P, g.stellar


SIZES = [(n, "sphere") for n in (1, 2, 16, 17, 64, 65, 1000, 1024, 1025, 2047, 16384, 16385, 32767, 32768, 32769, 50001)]
CASES = SIZES + [(n, k) for n in (300, 5000, 40000) for k in ("coincident", "all", "outlier", "nonfinite")]


@pytest.mark.parametrize("com", [0, 2])
@pytest.mark.parametrize("n,kind", CASES)
def test_fused_rebuild_equals_separate_kernels(gpu_lib, n, kind, com):
    P0, S0 = _case(n, kind)
    track = (n // 2, n - 1, [0.1, 0.2, 0.3], [1.0, 0.0, 0.0])
    other = ic.hernquist_sphere(100, 7)
    sim = NBodyGPU(0, P0, S0, walkGroup=32, walkSplit=1)
    pool = GalaxyPool(-(-n // 256) * 256 + 256, 2)
    slot = pool.add(P0, S0, KW, tracking=track)
    pool.add(other.particles, other.stellar, KW)
    sim.updateParams(**KW)
    sim.setTracking(*track)
    sim.setComMode(com)
    from galaxy_sim_b200._lib import check, lib
    check(lib().gs_set_com_mode(pool._ctx, com), pool._ctx)
    sim.sortBuild()
    pool.sort_build()
    for a, b in zip(sim.getTree(), pool.get_tree(slot)):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
    for a, b in zip(sim.readState(), pool.read_state(slot)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    if kind == "nonfinite":        # the forces are NaN; the rebuild is what is compared
        sim.destroy()
        pool.close()
        return
    sim.run(2, False)
    pool.run(2, False)
    for a, b in zip(sim.readState(), pool.read_state(slot)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(sim.getTracking(), pool.get_tracking(slot)):
        assert np.array_equal(a, b)
    assert sim.deviceErrors() == 0 and pool.device_errors(slot) == 0
    if n <= 32768:
        assert sim.stepKernels() == 3      # rebuild, walk, diagnostics
    sim.destroy()
    pool.close()
