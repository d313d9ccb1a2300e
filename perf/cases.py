"""The workloads whose speed this framework is judged by: whole steps of the
simulation in every mode a user runs, the FP64 accuracy reference and the
training of the learned acceptance criterion, all through the public classes.

A case is a dict of plain values:
  kind "step"    one BarnesHut.step of `n` bodies: `state` names the initial
                 conditions, `mac` the acceptance criterion, `mode` what close
                 pairs do, `form` the arithmetic form;
  kind "direct"  BarnesHut.direct_sum of `samples` bodies against all `n`;
  kind "train"   one epoch of BarnesHut.mac_train over `pairs` training pairs.
A step advances its state, so repeated passes are a running simulation; the
time steps are short enough that a state keeps its character over the passes
of a measurement.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import gravity_gb300
from gravity_gb300 import BarnesHut, abi, ic

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(gravity_gb300.__file__)), "mac_weights", "diverse.npy")


def _step(name, state, n, **kw):
    case = dict(name=name, kind="step", state=state, n=n, mac="plain", theta=0.5, softening=2.5e-5, dt=1e-3,
                mode="neither", form="fp32")
    case.update(kw)
    return case


def listed():
    return [
        # a small interactive scene: the step is launches and latency
        _step("plain_1k", "plummer", 1024, softening=1e-4),
        # the benchmark's small configuration, the reference's own rule
        _step("plain_65k", "plummer", 65536, softening=1e-4),
        # bouncing bodies in a wrapping box
        _step("collide_100k", "box", 100003, theta=0.7, softening=1e-4, dt=5e-5, mode="collision"),
        # a network-driven step of a mid-size state, ragged
        _step("learned_300k", "mixture", 299993, mac="learned", tolerance=-2.35),
        # the benchmark's merge configuration: static bounds, kills at the edge
        _step("merge_1m", "box", 1048576, theta=0.7, softening=1e-4, dt=5e-5, mode="merge"),
        # the encounter of two galaxies in the precision form
        _step("precision_2m", "galaxy", 2097152, form="precision"),
        # one decision per body group, no network needed
        _step("group_2m", "mixture", 2000003, mac="group"),
        # a large state under the reference's rule, ragged
        _step("plain_4m", "mixture", 4194301),
        # star clusters with merges under the learned rule
        _step("clusters_8m", "clusters", 8388608, mac="learned", tolerance=-2.4, dt=1e-4, mode="merge"),
        # the headline: the benchmark's largest learned step on one GPU
        _step("learned_16m", "mixture", 16777216, mac="learned", tolerance=-2.35),
        # the judge of every accuracy figure: an FP64 sum for sampled bodies
        dict(name="direct_1m", kind="direct", state="mixture", n=1048576, samples=4096, softening=2.5e-5),
        # one epoch of the criterion's training (forward, backward, Adam)
        dict(name="train_512k", kind="train", pairs=524288, batch=8192),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "group", "learned", "learned", "merge", "collide", "precision",
                       "clusters", "direct", "train"])
    if kind == "direct":
        return dict(kind="direct", state=rng.choice(["mixture", "plummer"]), n=_log_uniform(rng, 20000, 2000000),
                    samples=rng.randint(200, 4096), softening=2.5e-5)
    if kind == "train":
        return dict(kind="train", pairs=_log_uniform(rng, 20000, 1000000), batch=rng.choice([1000, 4096, 8192]))
    if kind == "collide":
        case = _step("", "box", _log_uniform(rng, 1000, 500000), theta=0.7, softening=1e-4, dt=5e-5, mode="collision")
    elif kind == "merge":
        case = _step("", "box", _log_uniform(rng, 1000, 2000000), theta=0.7, softening=1e-4, dt=5e-5, mode="merge")
    elif kind == "precision":
        case = _step("", rng.choice(["galaxy", "plummer"]), _log_uniform(rng, 2000, 3000000), form="precision")
    elif kind == "clusters":
        case = _step("", "clusters", _log_uniform(rng, 100000, 6000000), mac=rng.choice(["learned", "group"]),
                     tolerance=-2.4, dt=1e-4, mode=rng.choice(["merge", "neither"]))
    else:
        case = _step("", rng.choice(["plummer", "mixture", "galaxy"]), _log_uniform(rng, 1000, 5000000), mac=kind,
                     theta=round(rng.uniform(0.4, 0.8), 3), tolerance=round(rng.uniform(-2.6, -2.2), 3))
    del case["name"]
    return case


# ---- initial conditions, on the GPU, from the seed alone ------------------------


class _Rng:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def directions(self, n):
        d = self.normal(n, 3)
        return d / d.norm(dim=1, keepdim=True)


def _plummer(r, n):
    """Plummer sphere with unit mass and scale, isotropic speeds from its
    distribution function g(q) = q^2 (1 - q^2)^3.5 (inverted on a table)."""
    x = r.uniform(1e-10, 0.999, n)
    rad = (x.pow(-2.0 / 3.0) - 1.0).rsqrt()
    q = torch.linspace(0.0, 1.0, 4097, device="cuda", dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1.0 - q * q).clamp(min=0.0) ** 3.5, 0)
    at = torch.searchsorted(cdf / cdf[-1], r.uniform(0.0, 1.0, n)).clamp(max=4096)
    vesc = math.sqrt(2.0) * (1.0 + rad * rad) ** -0.25
    return r.directions(n) * rad[:, None], r.directions(n) * (q[at] * vesc)[:, None]


def _galaxy(r, n):
    """80% exponential disk, 20% Hernquist bulge, unit mass, near-circular."""
    nd = int(round(0.8 * n))
    R = -torch.log(r.uniform(1e-12, 1.0, nd) * r.uniform(1e-12, 1.0, nd))
    phi = r.uniform(0.0, 2.0 * math.pi, nd)
    z = -0.1 * torch.log(r.uniform(1e-12, 1.0, nd)) * torch.sign(r.uniform(-1.0, 1.0, nd))
    s = r.uniform(0.0, 0.999, n - nd).sqrt()
    rb = 0.2 * s / (1.0 - s)

    def enclosed(d):
        return 0.8 * (1.0 - torch.exp(-d) * (1.0 + d)) + 0.2 * d * d / (d + 0.2) ** 2

    vc = (enclosed(R) / R.clamp(min=1e-3)).sqrt()
    pos = torch.cat([torch.stack([R * phi.cos(), R * phi.sin(), z], 1), r.directions(n - nd) * rb[:, None]])
    vd = torch.stack([-vc * phi.sin(), vc * phi.cos(), torch.zeros_like(vc)], 1) + 0.05 * vc[:, None] * r.normal(nd, 3)
    vb = r.normal(n - nd, 3) * (enclosed(rb) / (3.0 * rb.clamp(min=1e-3))).sqrt()[:, None]
    return pos, torch.cat([vd, vb])


def _bodies(case, seed):
    """float32[n, 8] on the GPU: x, y, z, mass, vx, vy, vz, density."""
    r, n, state = _Rng(seed), case["n"], case["state"]
    out = torch.empty((n, 8), device="cuda", dtype=torch.float32)
    out[:, 7] = 1.0
    if state == "plummer":
        pos, vel = _plummer(r, n)
        out[:, 3] = 1.0 / n
    elif state == "mixture":  # 70% Plummer sphere in 30% resting field bodies
        k = int(round(0.7 * n))
        p, v = _plummer(r, k)
        pos = torch.cat([p, r.uniform(-3.0, 3.0, n - k, 3)])
        vel = torch.cat([v, torch.zeros((n - k, 3), device="cuda", dtype=torch.float64)])
        mix = torch.randperm(n, generator=r.g, device="cuda")
        pos, vel = pos[mix], vel[mix]
        out[:, 3] = 1.0 / n
    elif state == "galaxy":  # two disks on an encounter orbit
        k = n // 2
        (p1, v1), (p2, v2) = _galaxy(r, k), _galaxy(r, n - k)
        c, s = math.cos(math.pi / 3), math.sin(math.pi / 3)
        tilt = torch.tensor([[1.0, 0.0, 0.0], [0.0, c, s], [0.0, -s, c]], device="cuda", dtype=torch.float64)
        at = torch.tensor([5.0, 0.0, 0.0], device="cuda", dtype=torch.float64)
        by = torch.tensor([-0.29, 0.12, 0.0], device="cuda", dtype=torch.float64)
        pos, vel = torch.cat([p1 - at, p2 @ tilt + at]), torch.cat([v1 - by, v2 @ tilt + by])
        out[:, 3] = 2.0 / n
    elif state == "box":  # bodies with radii 2e-4 to 2e-3 in a cube
        pos = r.uniform(-1.0, 1.0, n, 3)
        vel = 0.1 * r.normal(n, 3) if case["mode"] == "collision" else torch.zeros_like(pos)
        out[:, 3] = 10.0 ** r.uniform(-6.0, -3.0, n)
        out[:, 7] = ic.MERGE_DENSITY
    else:  # 256 resting clusters, masses m^-2
        centre = r.uniform(-10.0, 10.0, 256, 3)
        sigma = 10.0 ** r.uniform(-2.0, -1.0, 256)
        which = torch.randint(0, 256, (n,), generator=r.g, device="cuda")
        pos = centre[which] + r.normal(n, 3) * sigma[which][:, None]
        vel = torch.zeros_like(pos)
        out[:, 3] = 1.0 / (1e9 - r.uniform(0.0, 1.0, n) * (1e9 - 1e6))
        out[:, 7] = ic.MERGE_DENSITY
    out[:, 0:3] = pos
    out[:, 4:7] = vel
    return out


# ---- the measured calls ---------------------------------------------------------

_MODES = {"neither": abi.MODE_NEITHER, "merge": abi.MODE_MERGE, "collision": abi.MODE_COLLISION}
_MACS = {"plain": abi.MAC_PLAIN, "learned": abi.MAC_LEARNED, "group": abi.MAC_GROUP}


def _simulation(bodies, bounds):
    host = bodies.cpu().numpy().reshape(-1).view(abi.BODY_DTYPE)
    sim = BarnesHut(len(host), bounds, abi.units(G=1.0))
    sim.upload_bodies(host)
    sim.init()
    return sim


def _exact_bounds(bodies):
    return torch.cat([bodies[:, :3].amin(0), bodies[:, :3].amax(0)]).cpu().numpy()


class _DeviceBodies:
    """The simulation's device body buffer as float32[n, 8], without a copy."""

    def __init__(self, sim, ptr):
        self.sim = sim  # the buffer lives as long as the simulation
        self.__cuda_array_interface__ = dict(shape=(sim.n, 8), typestr="<f4", data=(ptr, False), version=3, strides=None)


def prepare(case, seed):
    if case["kind"] == "train":
        r, m = _Rng(seed), case["pairs"]
        feats = r.uniform(-1.0, 1.0, m, abi.MAC_FEATURES)
        labels = -3.0 + feats @ r.uniform(-1.0, 1.0, abi.MAC_FEATURES) + (feats[:, 0] * feats[:, 1]) + 0.1 * r.normal(m)
        sim = BarnesHut(1024, [-1, -1, -1, 1, 1, 1], abi.units(G=1.0))
        sim.mac_set_weights(np.load(WEIGHTS))
        sim.mac_write_pairs(feats.float().cpu().numpy(), labels.float().cpu().numpy())
        return dict(kind="train", sim=sim, batch=case["batch"], seed=int(seed) & 0xFFFF)
    bodies = _bodies(case, seed)
    if case["kind"] == "direct":
        return dict(kind="direct", sim=_simulation(bodies, _exact_bounds(bodies)),
                    params=abi.step_params(softening=case["softening"]), sample=_sample(case, seed))
    static = case["state"] == "box"
    sim = _simulation(bodies, [-2, -2, -2, 2, 2, 2] if static else _exact_bounds(bodies))
    if case["mac"] == "learned":
        sim.mac_set_weights(np.load(WEIGHTS))
    params = abi.step_params(
        dt=case["dt"], theta=case["theta"], softening=case["softening"], mode=_MODES[case["mode"]],
        bounds=abi.BOUNDS_STATIC if static else abi.BOUNDS_DYNAMIC, wrap=case["mode"] == "collision", elasticity=0.5,
        mac=_MACS[case["mac"]], mac_tolerance=case.get("tolerance", -3.0),
        precision=abi.PRECISION_COMPENSATED if case["form"] == "precision" else abi.PRECISION_FP32)
    return dict(kind="step", sim=sim, params=params, views={})


def _sample(case, seed):
    pick = np.random.default_rng(int(seed)).choice(case["n"], case["samples"], replace=False)
    return np.sort(pick).astype(np.uint32)


def run(state):
    sim = state["sim"]
    if state["kind"] == "train":
        losses = sim.mac_train(1, batch=state["batch"], lr=1e-3, seed=state["seed"])
        return dict(losses=losses, weights=sim.mac_get_weights())
    if state["kind"] == "direct":
        return sim.direct_sum(state["params"], state["sample"])
    sim.step(state["params"])
    ptr = sim.device_ptrs().bodies_in  # the new state; steps alternate between two buffers
    out = state["views"].get(ptr)
    if out is None:
        b = torch.as_tensor(_DeviceBodies(sim, ptr), device="cuda")
        out = state["views"][ptr] = dict(pos_mass=b[:, :4], vel_density=b[:, 4:])
    return out


def work(case):
    if case["kind"] == "train":
        # features and label of each pair; forward, backward by weights and by
        # activations of the 12-32-32-1 network
        return dict(bytes=52 * case["pairs"], flops=3 * 2880 * case["pairs"])
    n = case["n"]
    if case["kind"] == "direct":
        return dict(bytes=16 * n + 28 * case["samples"], flops=20 * n * case["samples"])
    # bodies in and out, the leaf and internal nodes that the step publishes;
    # about 15 log2 n interactions of 20 flops per body at theta 0.5
    theta = case["theta"] if case["mac"] != "learned" else 0.5
    return dict(bytes=(32 + 32 + 160) * n, flops=20 * n * 15 * math.log2(n) * (0.5 / theta) ** 2)


# ---- the same in 64 bits, without this package's code ------------------------------


def _gravity64(target, bodies, soft):
    """Accelerations at `target` rows (indices) from all bodies, G = 1."""
    src = bodies.double()
    mass = src[:, 3].contiguous()
    xyz = [src[:, k].contiguous() for k in range(3)]
    out = torch.empty((len(target), 3), device="cuda", dtype=torch.float64)
    rows = max(1, (1 << 26) // len(bodies))
    for s in range(0, len(target), rows):
        t = target[s : s + rows]
        d = [x[None, :] - x[t][:, None] for x in xyz]
        w = mass * (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + soft).pow(-1.5)
        for k in range(3):
            out[s : s + rows, k] = (w * d[k]).sum(1)
    return out


def exact(case, seed):
    if case["kind"] == "train" or case["n"] * case.get("samples", case["n"]) > 1e11:
        return None
    bodies = _bodies(case, seed)
    soft = float(np.float32(case["softening"]))
    if case["kind"] == "direct":
        return _gravity64(torch.from_numpy(_sample(case, seed).astype(np.int64)).cuda(), bodies, soft).cpu().numpy()
    if case["mode"] != "neither":
        return None  # contacts are resolved in an order that a formula does not give
    dt = float(np.float32(case["dt"]))
    b = bodies.double()
    vel = b[:, 4:7] + dt * _gravity64(torch.arange(case["n"], device="cuda"), bodies, soft)
    return dict(pos_mass=torch.cat([b[:, :3] + dt * vel, b[:, 3:4]], 1), vel_density=torch.cat([vel, b[:, 7:8]], 1))
