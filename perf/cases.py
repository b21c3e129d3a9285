"""The work that a user of this package has it do, as measurable cases.

Kinds of case (the "kind" of a case dict):

* step:    one full time step of a lone galaxy from a state held on the GPU:
           Params upload, then codes + sort + gather + tree build + walk +
           kick-drift (+ star formation) through ``NBodyGPU.run(1)``. The state
           comes through the position and stellar buffers, as it does from an
           earlier step or from another device program.
* pool:    the same step for many galaxies of mixed sizes in one ``GalaxyPool``.
* frame:   one frame of an interactive viewer: Params upload, rebuild, step, star
           formation and the asynchronous position readback into host memory.
* refresh: the reference's own frame, a tree that stays for many steps: COM refresh
           of an uploaded tree from the current positions, then the step.
* sort:    the ``mortonTree.js`` bootstrap, host arrays in and out (``sortAndBuild``).

Galaxies are the package's seeded disks (gas with drag and star formation, or none),
two-disk collisions with tracked halo centres and Hernquist spheres, with the
masses, softenings, opening angles and time step of its workloads.
"""
import ctypes as C
import math

import numpy as np
import torch

from galaxy_sim_b200 import initial_conditions as ic
from galaxy_sim_b200._lib import check, lib
from galaxy_sim_b200.morton_tree import sortAndBuild
from galaxy_sim_b200.nbody_gpu import NBodyGPU
from galaxy_sim_b200.pool import GalaxyPool

DT = 0.005
TIME = 2.5          # simulation time of the step (it seeds star formation)
AGING = 25.0


def _step(name, n, preset="disk", theta=0.5, eps=0.02, gas=False, comp=False, com64=False):
    return {"name": name, "kind": "step", "n": n, "preset": preset, "theta": theta, "eps": eps, "gas": gas,
            "comp": comp, "com64": com64}


def listed():
    return [
        # the smallest galaxy of the batch and serving ranges, alone: launches and latency
        _step("step_disk_4k", 4096),
        # one disk of 16384, the small benchmark configuration
        _step("step_disk_16k", 16384, eps=0.05),
        # a ragged mid-size gas disk at the wider opening angle
        _step("step_gas_60001", 60001, theta=0.7, gas=True),
        # a ragged sphere at the wider angle with both precision options on
        _step("step_sphere_200003", 200003, preset="sphere", theta=0.7, eps=0.05, comp=True, com64=True),
        # the flagship: one disk of 524288 with gas drag and star formation
        _step("step_gas_512k", 524288, gas=True),
        # two disks of 262144 on a parabolic orbit, halo centres tracked
        _step("step_collision_512k", 524288, preset="collision"),
        # the largest served request
        _step("step_disk_1m", 1048576),
        # an ensemble in one pool, N log-uniform in [4096, 262144], some with gas
        {"name": "pool_16", "kind": "pool", "galaxies": 16, "nmin": 4096, "nmax": 262144, "sizes": 7,
         "theta": 0.5, "eps": 0.02},
        # the reference's interactive size: every frame's positions reach the host
        {"name": "frame_25000", "kind": "frame", "n": 25000, "theta": 0.5, "eps": 0.05, "gas": True},
        # the reference's frame loop between two tree swaps
        {"name": "refresh_step_100k", "kind": "refresh", "n": 100000, "theta": 0.5, "eps": 0.02},
        # the bootstrap sort and build of mortonTree.js
        {"name": "sort_and_build_100k", "kind": "sort", "n": 100000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "pool", "frame", "refresh", "sort"])
    theta = round(rng.uniform(0.5, 0.9), 3)
    eps = round(math.exp(rng.uniform(math.log(0.02), math.log(0.08))), 4)
    if kind == "step":
        preset = rng.choice(["disk", "disk", "sphere", "collision"])
        c = _step(None, _log_uniform(rng, 1000, 900000), preset, theta, eps,
                  gas=preset == "disk" and rng.random() < 0.5, comp=rng.random() < 0.2, com64=rng.random() < 0.2)
        del c["name"]
        return c
    if kind == "pool":
        return {"kind": "pool", "galaxies": rng.randint(2, 16), "nmin": 2000, "nmax": _log_uniform(rng, 20000, 262144),
                "sizes": rng.randint(1, 10 ** 6), "theta": theta, "eps": eps}
    if kind == "frame":
        return {"kind": "frame", "n": _log_uniform(rng, 2000, 100000), "theta": theta, "eps": eps,
                "gas": rng.random() < 0.5}
    if kind == "refresh":
        return {"kind": "refresh", "n": _log_uniform(rng, 2000, 400000), "theta": theta, "eps": eps}
    return {"kind": "sort", "n": _log_uniform(rng, 1000, 400000)}


# ---- inputs ------------------------------------------------------------------------------

def _galaxy(preset, n, seed, gas=False):
    if preset == "collision":
        return ic.two_galaxy_collision(n, seed, Q=1.5, arms=2, gas_frac=0.0)
    if preset == "sphere":
        return ic.hernquist_sphere(n, seed)
    return ic.galaxy_disk(n, seed, Q=1.2, arms=4, gas_frac=0.3 if gas else 0.0)


def _params(g, case, gas):
    return dict(dt=DT, G=1.0, epsilon=case["eps"], theta=case["theta"],
                haloMass=g.halo_mass if g.halo_centers else 0.0, haloA=g.halo_a, gasDrag=0.25 if gas else 0.0,
                time=TIME, agingRate=AGING, sfDensity=g.sf_density, sfEff=0.02 if gas else 0.0, sfDt=DT,
                haloCenters=[list(c) + [0.0] for c in g.halo_centers[:2]])


def _pool_members(case, seed):
    rng = np.random.default_rng(case["sizes"])
    out = []
    for k in range(case["galaxies"]):
        n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        gas = bool(rng.random() < 0.5)
        out.append((_galaxy("disk", n, 1000 * seed + k, gas), gas))
    return out


def _drifted(P):
    """The sorted records a fraction of a step later: the state a kept tree is refreshed from."""
    P = P.copy()
    P[:, :3] += np.float32(0.5 * DT) * P[:, 4:7]
    return P


class _DeviceMemory:
    """A device pointer as an array torch can view (float32). torch keeps this object as
    long as a view lives, and with it the context that owns the memory."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (pointer, False), "version": 3}


class _Views:
    """torch views of a context's ping-pong buffers, made once per buffer."""

    def __init__(self, owner):
        self.owner, self.made = owner, {}

    def of(self, pointer, shape):
        v = self.made.get(pointer)
        if v is None:
            v = self.made[pointer] = torch.as_tensor(_DeviceMemory(self.owner, pointer, shape), device="cuda")
        return v


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    kind = case["kind"]
    if kind == "sort":
        g = _galaxy("disk", case["n"], seed, True)
        s.particles, s.stellar = g.particles, g.stellar
        return s
    if kind == "pool":
        members = _pool_members(case, seed)
        s.pool = GalaxyPool(sum(-(-g.N // 256) * 256 for g, _ in members), len(members))
        s.members = []
        for g, gas in members:
            p = _params(g, case, gas)
            slot = s.pool.add(g.particles, g.stellar, p, star_formation=gas)
            s.members.append((slot, g.N, p, torch.from_numpy(g.particles).cuda(), torch.from_numpy(g.stellar).cuda()))
        s.views, s.stream = _Views(s.pool), torch.cuda.ExternalStream(s.pool.stream)
        return s
    gas = bool(case.get("gas"))
    g = _galaxy(case.get("preset", "disk"), case["n"], seed, gas)
    s.params, s.gas = _params(g, case, gas), gas
    s.tracking = (g.central, g.halo_centers) if case.get("preset") == "collision" else None
    particles, stellar = g.particles, g.stellar
    if kind == "refresh":
        built = sortAndBuild(particles, stellar, g.N)
        particles, stellar = built["sorted"].reshape(-1, 8), built["sortedStellar"].reshape(-1, 4)
    s.gpu = NBodyGPU(0, particles, stellar)
    s.n = g.N
    if kind == "refresh":
        tree = built["tree"]
        s.gpu.uploadBHTree(tree.nodes, tree.numNodes, tree.levelRanges)
        particles = _drifted(particles)
    if case.get("comp"):
        s.gpu.setWalkMode(True)
    if case.get("com64"):
        s.gpu.setComMode(2)
    s.particles, s.stellar = torch.from_numpy(particles).cuda(), torch.from_numpy(stellar).cuda()
    s.views, s.stream = _Views(s.gpu), torch.cuda.ExternalStream(s.gpu.stream)
    if kind == "frame":
        s.staging = torch.empty(4 * s.n, dtype=torch.float32, pin_memory=True).numpy()
    return s


def _records(v):
    return {"position": v[:, :4], "velocity": v[:, 4:7], "pad": v[:, 7]}


def run(state):
    """One pass. The context's stream follows the caller's current stream and the caller's
    stream follows it again, as for any program that goes on with the outputs."""
    if state.case["kind"] == "sort":
        return _sort(state)
    here = torch.cuda.current_stream()
    state.stream.wait_stream(here)
    out = (_pool if state.case["kind"] == "pool" else _lone)(state)
    here.wait_stream(state.stream)
    return out


def _sort(s):
    r = sortAndBuild(s.particles, s.stellar, s.case["n"], 1)
    tree = r["tree"]
    words, reals = tree.i32.reshape(-1, 16), tree.f32.reshape(-1, 16)   # the whole node pool
    return {"sorted": r["sorted"], "sortedStellar": r["sortedStellar"], "perm": r["perm"].view(np.int32),
            "masses": r["masses"], "central": [r["centralIdx"], r["centralIdx2"]],
            "nodes": tree.numNodes, "com": reals[:, :3], "mass": reals[:, 3], "size": reals[:, 4],
            "links": words[:, 5:]}


def _pool(s):
    pool, L, views, out, d = s.pool, lib(), s.views, [], C.c_void_p()
    with torch.cuda.stream(s.stream):
        for slot, n, params, particles, stellar in s.members:
            pool.set_params(slot, **params)      # selects the galaxy too
            check(L.gs_position_buffer(pool._ctx, C.byref(d)), pool._ctx)
            views.of(d.value, (n, 8)).copy_(particles)
            check(L.gs_stellar_buffer(pool._ctx, C.byref(d)), pool._ctx)
            views.of(d.value, (n, 4)).copy_(stellar)
    pool.run(1, True)
    for slot, n, _, _, _ in s.members:
        check(L.gs_select(pool._ctx, slot), pool._ctx)
        check(L.gs_position_buffer(pool._ctx, C.byref(d)), pool._ctx)
        r = _records(views.of(d.value, (n, 8)))
        check(L.gs_stellar_buffer(pool._ctx, C.byref(d)), pool._ctx)
        out.append([r["position"], r["velocity"], views.of(d.value, (n, 4))])
    return out


def _lone(s):
    kind, gpu, n, views = s.case["kind"], s.gpu, s.n, s.views
    gpu.updateParams(**s.params)
    with torch.cuda.stream(s.stream):
        views.of(gpu.positionBuffer, (n, 8)).copy_(s.particles)
        views.of(gpu.stellarBuffer, (n, 4)).copy_(s.stellar)
    if kind == "frame":
        gpu.sortBuild()
        gpu.step()
        if s.gas:
            gpu.encodeStarFormation()
        gpu.encodePositionReadback(staging=s.staging)
        return {"positions": gpu.readPositions().reshape(n, 4), "stellar": views.of(gpu.stellarBuffer, (n, 4))}
    if kind == "refresh":
        gpu.encodeRefresh()
        gpu.step()
        return _records(views.of(gpu.positionBuffer, (n, 8)))
    if s.tracking is not None:
        (c1, c2), centres = s.tracking
        gpu.setTracking(c1, c2, centres[0], centres[1])
    gpu.run(1, s.gas)
    return dict(_records(views.of(gpu.positionBuffer, (n, 8))), stellar=views.of(gpu.stellarBuffer, (n, 4)))


# ---- what a pass cannot do without ----------------------------------------------------------

def _interactions(n, theta):
    """Interactions per particle of these disks (monopoles + leaf pairs) under the acceptance
    rule: about 1070 at 524288 particles and an opening angle of 0.5, growing with log n."""
    return 1070.0 * (0.5 / theta) ** 2.26 * max(0.1, math.log2(max(n, 2) / 64.0) / 13.0)


def work(case):
    if case["kind"] == "sort":      # records in and out, permutation, masses, 64-byte nodes
        return {"bytes": case["n"] * (48 + 48 + 4 + 4 + 0.25 * 64), "flops": 0.0}
    if case["kind"] == "pool":
        rng = np.random.default_rng(case["sizes"])
        ns = []
        for _ in range(case["galaxies"]):
            ns.append(int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]))))))
            rng.random()
    else:
        ns = [case["n"]]
    record = {"step": 96, "pool": 96, "frame": 112, "refresh": 64}[case["kind"]]
    return {"bytes": float(sum(n * record for n in ns)),
            "flops": float(sum(23.0 * n * _interactions(n, case["theta"]) for n in ns))}


# ---- the same in 64 bits ----------------------------------------------------------------------

def _interleave(q):
    v = q & 0x3ff
    v = (v | (v << 16)) & 0x30000ff
    v = (v | (v << 8)) & 0x300f00f
    v = (v | (v << 4)) & 0x30c30c3
    return (v | (v << 2)) & 0x9249249


def _codes(x):
    """30-bit Morton codes and the root cube's size of float64 positions (n, 3)."""
    lo = x.min(0).values
    size = float((x.max(0).values - lo).max()) * 1.0001 + 1e-9
    q = ((x - lo) * (1024.0 / size)).long().clamp(max=1023)
    return _interleave(q[:, 0]) | (_interleave(q[:, 1]) << 1) | (_interleave(q[:, 2]) << 2), size


def _levels(codes, size):
    """The bucketed octree over sorted codes, level by level: node ranges, leaf flags,
    each node's first child and child count (indices into the next level)."""
    n, dev = codes.numel(), codes.device
    start, end = torch.zeros(1, dtype=torch.long, device=dev), torch.full((1,), n, device=dev)
    levels = []
    for d in range(11):
        leaf = (end - start <= 16) | (d == 10)
        lv = {"start": start, "end": end, "leaf": leaf, "size": size * 0.5 ** d,
              "child": torch.zeros_like(start), "children": torch.zeros_like(start)}
        levels.append(lv)
        inner = torch.nonzero(~leaf).flatten()
        if not inner.numel():
            break
        step = torch.zeros(n + 1, dtype=torch.long, device=dev)
        step[start[inner]] += 1
        step.index_add_(0, end[inner], torch.full_like(inner, -1))
        prefix = codes >> (27 - 3 * d)
        first = torch.ones(n, dtype=torch.bool, device=dev)
        first[1:] = prefix[1:] != prefix[:-1]
        child = torch.nonzero(first & (step.cumsum(0)[:n] > 0)).flatten()
        parent = inner[torch.searchsorted(start[inner], child, right=True) - 1]
        after = torch.cat([child[1:], torch.full((1,), n, device=dev)])
        lv["children"].index_add_(0, parent, torch.ones_like(parent))
        lv["child"] = lv["children"].cumsum(0) - lv["children"]
        start, end = child, torch.minimum(after, end[parent])
    return levels


def _moments(levels, x, m):
    """Mass and centre of mass of every node."""
    i = torch.arange(x.shape[0], device=x.device)
    for lv in levels:
        k = torch.searchsorted(lv["start"], i, right=True) - 1
        inside = (k >= 0) & (i < lv["end"][k.clamp(min=0)])
        k, j = k[inside], i[inside]
        mass = torch.zeros(lv["start"].numel(), dtype=torch.float64, device=x.device).index_add_(0, k, m[j])
        mx = torch.zeros(mass.numel(), 3, dtype=torch.float64, device=x.device).index_add_(0, k, m[j, None] * x[j])
        lv["mass"] = mass
        lv["com"] = torch.where(mass[:, None] > 0, mx / mass[:, None], torch.zeros_like(mx))


def _expand(first, count):
    """(owner, value) of the concatenated ranges [first, first + count)."""
    owner = torch.repeat_interleave(torch.arange(first.numel(), device=first.device), count)
    at = torch.arange(owner.numel(), device=first.device) - (count.cumsum(0) - count)[owner]
    return owner, first[owner] + at


def _walk(levels, x, m, theta, eps2):
    """Acceleration and potential (G = 1) and own-leaf density of every particle."""
    n, dev = x.shape[0], x.device
    acc = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    pot = torch.zeros(n, dtype=torch.float64, device=dev)
    dens = torch.zeros(n, dtype=torch.float64, device=dev)

    def add(p, r, mass, d2):
        inv = d2.rsqrt()
        acc.index_add_(0, p, (mass * inv ** 3)[:, None] * r)
        pot.index_add_(0, p, -mass * inv)

    for c0 in range(0, n, 32768):
        p = torch.arange(c0, min(n, c0 + 32768), device=dev)
        k = torch.zeros_like(p)
        for lv in levels:
            heavy = lv["mass"][k] != 0
            p, k = p[heavy], k[heavy]
            if not p.numel():
                break
            leaf, s2 = lv["leaf"][k], lv["size"] ** 2
            own = leaf & (p >= lv["start"][k]) & (p < lv["end"][k])
            dens[p[own]] = (lv["end"][k[own]] - lv["start"][k[own]]).double() / lv["size"] ** 3
            r = lv["com"][k] - x[p]
            d2 = (r * r).sum(1) + eps2
            far = (s2 < theta * theta * d2) if s2 >= 0.25 * eps2 else torch.ones_like(leaf)
            add(p[far], r[far], lv["mass"][k[far]], d2[far])
            near = leaf & ~far
            pn, kn = p[near], k[near]
            owner, j = _expand(lv["start"][kn], lv["end"][kn] - lv["start"][kn])
            i = pn[owner]
            other = i != j
            i, j = i[other], j[other]
            r = x[j] - x[i]
            add(i, r, m[j], (r * r).sum(1) + eps2)
            opened = ~leaf & ~far
            owner, child = _expand(lv["child"][k[opened]], lv["children"][k[opened]])
            p, k = p[opened][owner], child
    return acc, pot, dens


def _f32(v):
    return float(np.float32(v))


def _advance(P, params, tree=None):
    """One step of float32 records P (n, 8), in the order of the sort (or with the given sorted
    records' tree): positions, velocities, pads and the energies of the diagnostics."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    P = torch.as_tensor(P, device=dev).double()
    if tree is None:
        codes, size = _codes(P[:, :3])
        order = torch.argsort(codes, stable=True)
        P, codes = P[order], codes[order]
    else:
        codes, size = _codes(torch.as_tensor(tree, device=dev).double()[:, :3])
    x, m, v, gas = P[:, :3].contiguous(), P[:, 3].contiguous(), P[:, 4:7], P[:, 7] < -0.5
    levels = _levels(codes, size)
    _moments(levels, x, m)
    acc, pot, dens = _walk(levels, x, m, _f32(params["theta"]), _f32(float(params["epsilon"]) ** 2))
    dt, hm, ha = _f32(params["dt"]), _f32(params["haloMass"]), _f32(params["haloA"])
    halo = torch.zeros_like(pot)
    if hm > 0:
        for c in params["haloCenters"]:
            d = x - torch.tensor([_f32(q) for q in c[:3]], dtype=torch.float64, device=dev)
            r = d.norm(dim=1).clamp(min=1e-6)
            acc = acc - d * (hm / ((r + ha) ** 2 * r))[:, None]
            halo = halo - hm / (r + ha)
    v = v + acc * dt
    if params["gasDrag"] > 0:
        u = torch.stack([-x[:, 1], x[:, 0], torch.full_like(pot, 1e-6)], 1)
        u = u / u.norm(dim=1, keepdim=True)
        along = (v * u).sum(1, keepdim=True) * u
        v = torch.where(gas[:, None], along + (v - along) * math.exp(-_f32(params["gasDrag"]) * dt), v)
    e = 0.5 * (v * v).sum(1) + 0.5 * pot + halo
    return {"position": torch.cat([x + v * dt, m[:, None]], 1), "velocity": v,
            "pad": torch.where(gas, -(1.0 + dens), torch.zeros_like(dens)), "energy": e}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = _galaxy("disk", case["n"], seed, True)
        P = torch.from_numpy(g.particles).double()
        codes, size = _codes(P[:, :3])
        order = torch.argsort(codes, stable=True)
        levels = _levels(codes[order], size)
        _moments(levels, P[order, :3].contiguous(), P[order, 3].contiguous())
        sizes = [torch.full((lv["start"].numel(),), lv["size"], dtype=torch.float64) for lv in levels]

        def pool(parts):
            v = torch.cat(parts)
            return torch.cat([v, torch.zeros((2 * g.N + 4096 - v.shape[0],) + v.shape[1:], dtype=v.dtype)])

        return {"sorted": P[order].flatten(), "sortedStellar": torch.from_numpy(g.stellar).double()[order].flatten(),
                "perm": None, "masses": P[order, 3], "central": [None, None],
                "nodes": None, "com": pool([lv["com"] for lv in levels]), "mass": pool([lv["mass"] for lv in levels]),
                "size": pool(sizes), "links": None}
    if kind == "pool":
        out = []
        for g, gas in _pool_members(case, seed):
            r = _advance(g.particles, _params(g, case, gas))
            out.append([r["position"], None if gas else r["velocity"], None])
        return out
    gas = bool(case.get("gas"))
    g = _galaxy(case.get("preset", "disk"), case["n"], seed, gas)
    params = _params(g, case, gas)
    if kind == "refresh":
        P = torch.from_numpy(g.particles)
        P = P[torch.argsort(_codes(P[:, :3].double())[0], stable=True)].numpy()
        r = _advance(_drifted(P), params, tree=P)
        return {k: r[k] for k in ("position", "velocity", "pad")}
    r = _advance(g.particles, params)
    if kind == "frame":
        return {"positions": torch.cat([r["position"][:, :3], r["energy"][:, None]], 1), "stellar": None}
    # star formation changes a few velocities and pads after the step
    return {"position": r["position"], "velocity": None if gas else r["velocity"], "pad": None if gas else r["pad"],
            "stellar": None}
