"""Walks over states with non-finite positions: a particle at a NaN position fails every
compare of the opening test, so it opens every node it meets, but no node twice and none
outside its galaxy's tree. Interaction counts equal the FP64 walk of the same rule, the
device error word says GS_DERR_TREE (the empty slots of a staged range were opened), and
particles whose walk meets no non-finite value, and the other galaxies of a pool, are
not touched. Every walk group size, with and without splits.

Tolerance: counts may differ by an acceptance decision on the very edge that falls the
other way in FP32 (1e-4 of them, as for finite states); everything else is compared bit
for bit."""
import numpy as np
import pytest

from galaxy_sim_b200 import _lib
from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200.nbody_gpu import NBodyGPU
from galaxy_sim_b200.pool import GalaxyPool

pytestmark = pytest.mark.gpu

KW = dict(dt=0.005, G=1.0, epsilon=1e-3, theta=0.5)
SETTINGS = [(32, 1), (16, 1), (16, 2), (8, 1), (8, 4), (4, 8)]


@pytest.mark.parametrize("group,split", SETTINGS)
@pytest.mark.parametrize("n,kind", [(2, "one"), (33, "one"), (300, "one"), (3001, "one"), (3001, "inf"), (17, "all"),
                                    (300, "all"), (3001, "all")])
def test_counts_equal_the_fp64_walk(gpu_lib, oracle, n, kind, group, split):
    P0 = ic.hernquist_sphere(n, 70 + n).particles.copy()
    if kind == "one":
        P0[n // 2, 1] = np.nan
    elif kind == "inf":
        P0[n // 2, 0] = np.inf
    else:
        P0[:, :3] = np.nan
    sim = NBodyGPU(0, P0, walkGroup=group, walkSplit=split)
    sim.updateParams(**dict(KW, dt=0.0))
    sim.setDebug(True)
    sim.sortBuild()
    P, _ = sim.readState()
    nodes, lr, _ = sim.getTree()
    sim.counters(reset=True)
    sim.step()
    err = sim.deviceErrors(clear=True)
    count = sim.counters()
    sim.destroy()
    p = oracle.make_params(n, epsilon=KW["epsilon"], theta=0.5, dt=0.0)
    _, _, _, want = oracle.walk_f64(p, P, nodes, oracle.refresh_f64(P, nodes, lr))
    for k in range(3):
        assert abs(count[k] - int(want[k])) <= 1e-4 * int(want[k]) + 16 * (kind != "all"), (k, count, want)
    if kind == "all":                # a chain of ten nodes and one leaf that holds every particle
        assert count == [0, n * (n - 1), n * len(nodes)]
    assert err == (0 if kind == "inf" else _lib.DERR_TREE)


@pytest.mark.parametrize("group,split", SETTINGS)
def test_a_lost_tracer_leaves_the_others_alone(gpu_lib, group, split):
    """Twenty massless tracers share a deepest cell, one of them at a NaN position: its leaf
    has no mass, so nobody else opens it, and every particle outside its own walk group of
    32 gets the bits it gets when the tracer is finite."""
    g = ic.hernquist_sphere(3000, 5)
    P0 = np.concatenate([np.zeros((20, 8), np.float32), g.particles])
    P0[:20, :3] = g.particles[:, :3].min(0)
    out = []
    for lost in (False, True):
        P = P0.copy()
        if lost:
            P[7, :3] = np.nan
        sim = NBodyGPU(0, P, walkGroup=group, walkSplit=split)
        sim.updateParams(**KW)
        sim.setDebug(True)
        sim.sortBuild()
        sim.step()
        assert sim.deviceErrors(clear=True) == (_lib.DERR_TREE if lost else 0)
        out.append((sim.readState()[0], *sim.readForces()))
        sim.destroy()
    for a, b in zip(*out):
        assert np.isfinite(a).all()
        assert np.array_equal(a[32:].view(np.uint32), b[32:].view(np.uint32))


@pytest.mark.parametrize("kind", ["one", "all", "coincident"])
def test_a_lost_galaxy_leaves_its_pool_alone(gpu_lib, kind):
    gs = [ic.hernquist_sphere(n, 80 + n) for n in (2000, 3001, 1500)]
    bad = gs[1].particles.copy()
    kw = dict(KW)
    if kind == "one":
        bad[1000, :3] = np.nan
    elif kind == "all":
        bad[:, :3] = np.nan
    else:                            # two particles at one place without softening: NaN after a step
        bad[1000, :3] = bad[1001, :3]
        kw["epsilon"] = 0.0
    pool = GalaxyPool(8192, 3)
    slots = [pool.add(gs[0].particles, gs[0].stellar, KW), pool.add(bad, gs[1].stellar, kw),
             pool.add(gs[2].particles, gs[2].stellar, KW)]
    pool.run(4, False)
    assert pool.device_errors(slots[1], clear=True) == _lib.DERR_TREE
    assert np.isnan(pool.read_state(slots[1])[0][:, :3]).any()
    for k in (0, 2):
        sim = NBodyGPU(0, gs[k].particles, gs[k].stellar, walkGroup=32, walkSplit=1)
        sim.updateParams(**KW)
        sim.run(4, False)
        assert np.array_equal(sim.readState()[0].view(np.uint32), pool.read_state(slots[k])[0].view(np.uint32))
        assert pool.device_errors(slots[k]) == 0
        sim.destroy()
    pool.close()


@pytest.mark.parametrize("group,split", SETTINGS)
@pytest.mark.parametrize("per", [12, 50])
def test_sizes_whose_squares_overflow(gpu_lib, oracle, per, group, split):
    """Two clumps 2e20 apart: size^2 of the upper nodes and r^2 between the clumps are +inf,
    such a node is never accepted, and the particles of a clump attract one another. The
    other clump's pull is 1e-18 of that and 0 in FP32; the rest are a few dozen terms
    summed in FP32."""
    P0 = np.zeros((2 * per, 8), np.float32)
    P0[:, 0] = np.repeat([-1e20, 1e20], per)
    P0[:, 1] = np.tile(np.arange(per) * 1e10, 2)
    P0[:, 3] = 1.0
    sim = NBodyGPU(0, P0, walkGroup=group, walkSplit=split)
    sim.updateParams(dt=0.0, G=1.0, epsilon=0.0, theta=0.5)
    sim.setDebug(True)
    sim.sortBuild()
    P, _ = sim.readState()
    nodes, lr, _ = sim.getTree()
    sim.step()
    assert sim.deviceErrors() == 0
    acc, _ = sim.readForces()
    sim.destroy()
    p = oracle.make_params(2 * per, epsilon=0.0, theta=0.5, dt=0.0)
    want, _, _, _ = oracle.walk_f64(p, P, nodes, oracle.refresh_f64(P, nodes, lr))
    assert np.all(np.abs(acc[:, 1] - want[:, 1]) <= 1e-5 * np.abs(want[:, 1]).max())
    assert np.abs(want[:, 1]).max() > 1e-20


@pytest.mark.parametrize("group,split", SETTINGS)
@pytest.mark.parametrize("n,far", [(5, None), (700, None), (700, 1e5), (700, 3e19)])
def test_zero_opening_angle_opens_every_node(gpu_lib, n, far, group, split):
    P0 = ic.hernquist_sphere(n, 90 + n).particles.copy()
    if far:
        P0[n // 3, 0] = far
    sim = NBodyGPU(0, P0, walkGroup=group, walkSplit=split)
    sim.updateParams(dt=0.0, G=1.0, epsilon=1e-3, theta=0.0)
    sim.setDebug(True)
    sim.sortBuild()
    nodes, _, _ = sim.getTree()
    sim.counters(reset=True)
    sim.step()
    assert sim.counters() == [0, n * (n - 1), n * len(nodes)]
    assert sim.deviceErrors() == 0
    sim.destroy()


@pytest.mark.parametrize("n", [300, 5000, 40000])
@pytest.mark.parametrize("kind", ["one", "inf", "all"])
def test_steps_equal_a_pools(gpu_lib, n, kind):
    """Full steps of such a galaxy alone (one rebuild kernel up to 32768 particles) and
    in a pool (separate rebuild kernels): the same finite values, NaNs at the same places,
    the same error word."""
    g = ic.hernquist_sphere(n, 60 + n)
    P0 = g.particles.copy()
    if kind == "all":
        P0[:, :3] = np.nan
    else:
        P0[n // 2, 0] = np.nan if kind == "one" else np.inf
    other = ic.hernquist_sphere(100, 7)
    sim = NBodyGPU(0, P0, g.stellar, walkGroup=32, walkSplit=1)
    pool = GalaxyPool(-(-n // 256) * 256 + 256, 2)
    slot, fine = pool.add(P0, g.stellar, KW), pool.add(other.particles, other.stellar, KW)
    sim.updateParams(**KW)
    sim.run(2, False)
    pool.run(2, False)
    err = sim.deviceErrors(clear=True)
    assert err == pool.device_errors(slot, clear=True) and pool.device_errors(fine) == 0
    for a, b in zip(sim.readState(), pool.read_state(slot)):
        assert np.array_equal(a, b, equal_nan=True)
    assert (sim.stepKernels() == 3) == (n <= 32768)
    sim.destroy()
    pool.close()
