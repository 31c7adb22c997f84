"""The engine's work, as a user's program calls for it: what is timed and compared.

A case is one call pattern of the public API (Simulation, Ensemble, Renderer)
with its sizes and options.  ``listed()`` gives fixed cases, ``draw(rng)`` more
of the same ranges; ``prepare`` builds what a program holds before the call,
``run`` makes one pass, ``work`` says what a pass cannot do without, and
``exact`` gives a pass's results from an FP64 direct sum in plain torch.

Kinds of pass
  step       one frame of a running simulation (the bodies stay on the GPU)
  restart    the initial state put back into the handle's buffers, then one frame
  roundtrip  upload of a state from page-locked host memory, one frame, download
  forces     accelerations at the current positions, to the host
  rollout    upload, differentiable rollout, gradients to the host
  render     one density frame and its tone-mapped image
  diagnose   the FP64 conserved quantities with the direct-sum potential
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

bh = importlib.import_module("webgpu-fluid-sim_b200")

# Option sets in use: the reference simulator's own settings, and the
# settings of the named workloads (webgpu-fluid-sim_b200/config.py) with the
# walk shapes their autotuner picks.
REFERENCE = dict(walk="exact", softening="reference", theta=0.6, dt=0.1 / 60.0, eps=1e-3, bits=32,
                 domain="fixed2000", integrator="symplectic-euler", leaf=1, bpl=2, multipole=2,
                 far=0.0)
DISKS = dict(REFERENCE, walk="group", softening="plummer", theta=0.5, dt=5e-5, domain="bbox",
             leaf=4, bpl=4, far=0.4)
EXACT_DISKS = dict(DISKS, walk="exact", leaf=1, bpl=2, far=0.0)
LEAPFROG = dict(DISKS, theta=0.7, dt=1e-4, integrator="leapfrog-kdk", leaf=8, bpl=2, far=0.0)
MIXTURE = dict(DISKS, dt=1e-5, eps=1e-4, bits=64, domain="fixed2000")
ENSEMBLE = dict(LEAPFROG, theta=0.5, leaf=4, far=0.4)
ROLLOUT = dict(LEAPFROG, theta=0.5, leaf=4)


def listed():
    return [
        # the reference's smallest scenes: launches and latency count
        dict(REFERENCE, name="frame-2k-exact", kind="restart", n=2000, scenario="two-clusters"),
        # the reference's default page: 50,000 bodies, default settings
        dict(REFERENCE, name="frame-50k-exact", kind="restart", n=50_000, scenario="default"),
        # the reference's walk at its UI's largest body count
        dict(EXACT_DISKS, name="step-800k-exact", kind="step", n=800_000,
             scenario="colliding-disks"),
        # a force evaluation at an odd size, read back
        dict(DISKS, name="forces-100k", kind="forces", n=100_003, scenario="plummer-projection",
             far=0.0),
        # the parity workload: leapfrog, group walk
        dict(LEAPFROG, name="step-16k-leapfrog", kind="step", n=16_384,
             scenario="uniform-disk-kepler"),
        # the headline workload
        dict(DISKS, name="step-800k", kind="step", n=800_000, scenario="colliding-disks"),
        # the largest workload: 64-bit keys, Gaussian mixture with duplicates
        dict(MIXTURE, name="step-16m-64bit", kind="step", n=16_777_216,
             scenario="gaussian-mixture"),
        # the headline workload driven from host memory, every step read back
        dict(DISKS, name="roundtrip-800k", kind="roundtrip", n=800_000,
             scenario="colliding-disks"),
        # a batch of independent systems of mixed sizes in one handle
        dict(ENSEMBLE, name="ensemble-64", kind="step", systems=64, lo=1024, hi=65_536),
        # optimising initial conditions: forward and backward through 20 steps
        dict(ROLLOUT, name="rollout-65k", kind="rollout", n=65_536, scenario="uniform-disk-kepler",
             steps=20, every=10),
        # one displayed frame of the headline workload
        dict(DISKS, name="render-800k-1080p", kind="render", n=800_000,
             scenario="colliding-disks", width=1920, height=1080, zoom=0.15),
        # one entry of the run log with the energy drift
        dict(DISKS, name="diagnose-200k", kind="diagnose", n=200_000, scenario="colliding-disks"),
    ]


def _size(rng, lo, hi):
    """Log-uniform whole size; one in four a multiple of 1024 where it fits."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if n >= 2048 and rng.random() < 0.25:
        n -= n % 1024
    return n


def draw(rng):
    disks = rng.choice(["colliding-disks", "uniform-disk-kepler", "plummer-projection"])
    kind = rng.choice(["restart", "step-exact", "step", "step", "step-64", "leapfrog", "forces",
                       "roundtrip", "ensemble", "rollout", "render", "diagnose"])
    group = dict(theta=rng.choice([0.4, 0.5, 0.6, 0.7]), leaf=rng.choice([2, 4, 8]),
                 bpl=rng.choice([1, 2, 4, 4]), multipole=rng.choice([2, 2, 2, 1]))
    group["far"] = 0.4 if group["multipole"] == 2 and rng.random() < 0.6 else 0.0
    if kind == "restart":
        return dict(REFERENCE, kind="restart", n=_size(rng, 1000, 200_000),
                    scenario=rng.choice(["default", "two-clusters", "planetary-disk"]))
    if kind == "step-exact":
        return dict(EXACT_DISKS, kind="step", n=_size(rng, 50_000, 800_000), scenario=disks,
                    theta=rng.choice([0.5, 0.6, 0.7]), leaf=rng.choice([1, 1, 8]))
    if kind == "step":
        return {**DISKS, **group, "kind": "step", "n": _size(rng, 4000, 1_500_000),
                "scenario": disks}
    if kind == "step-64":
        return {**MIXTURE, **group, "kind": "step", "n": _size(rng, 100_000, 6_000_000),
                "scenario": "gaussian-mixture"}
    if kind == "leapfrog":
        return {**LEAPFROG, **group, "kind": "step", "n": _size(rng, 4000, 400_000),
                "scenario": disks}
    if kind == "forces":
        case = {**DISKS, **group, "kind": "forces", "n": _size(rng, 1000, 400_000),
                "scenario": disks}
        if rng.random() < 0.3:
            case.update(walk="exact", far=0.0, leaf=1, softening=rng.choice(["plummer", "reference"]))
        return case
    if kind == "roundtrip":
        return dict(DISKS, kind="roundtrip", n=_size(rng, 10_000, 800_000), scenario=disks)
    if kind == "ensemble":
        return dict(ENSEMBLE, kind="step", systems=_size(rng, 4, 64), lo=_size(rng, 300, 4000),
                    hi=_size(rng, 8000, 65_536))
    if kind == "rollout":
        return dict(ROLLOUT, kind="rollout", n=_size(rng, 1000, 65_536), scenario=disks,
                    steps=rng.choice([5, 10, 20]), every=rng.choice([3, 5, 10]))
    if kind == "render":
        w, h = rng.choice([(640, 480), (1280, 720), (1920, 1080), (2560, 1440), (1001, 777)])
        return dict(DISKS, kind="render", n=_size(rng, 10_000, 800_000), width=w, height=h,
                    scenario=rng.choice([disks, disks, "default"]),
                    zoom=rng.choice([0.15, 0.5, 1.0]))
    return dict(DISKS, kind="diagnose", n=_size(rng, 10_000, 200_000), scenario=disks,
                softening=rng.choice(["plummer", "plummer", "reference"]))


class _Borrowed:
    """A device buffer of a handle, for torch; keeps the handle alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, version=2,
                                             data=(int(ptr), False))


def _view(owner, ptr, shape, typestr="<f4"):
    return torch.as_tensor(_Borrowed(owner, ptr, shape, typestr), device="cuda")


def _config(case):
    return bh.Config(bhTheta=case["theta"], deltaTime=case["dt"], softening=case["softening"],
                     plummerEps=case["eps"], mortonBits=case["bits"], mortonDomain=case["domain"],
                     integrator=case["integrator"], leafSize=case["leaf"], walk=case["walk"],
                     multipole=case["multipole"], bodiesPerLane=case["bpl"], farAlpha=case["far"])


def _simulation(case, seed):
    if "systems" in case:
        sizes = bh.ensemble_sizes(case["systems"], case["systems"], case["lo"], case["hi"])
        sim = bh.Ensemble(sizes, _config(case))
        sim.setScenarios(None, seed=seed)
        return sim
    sim = bh.Simulation(_config(case))
    if case["n"] > 1_000_000:  # generated on the GPU
        sim.setScenarioOnDevice(case["scenario"], seed)
        sim.setNumBodies(case["n"])
    else:
        sim.setNumBodies(case["n"])
        sim.setScenario(case["scenario"], seed)
    return sim


def prepare(case, seed):
    sim = _simulation(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, sim=sim)
    n = sim.getNumBodies()
    if kind in ("step", "restart"):
        b = sim.getBuffers()
        st["out"] = {"pos": _view(sim, b.pos, (n, 2)), "vel": _view(sim, b.vel, (n, 2))}
        if case["integrator"] == "leapfrog-kdk":
            st["out"]["acc"] = _view(sim, b.acc, (n, 2))
        if kind == "restart":
            torch.cuda.synchronize()
            st["start"] = {k: v.clone() for k, v in st["out"].items()}
            st["stream"] = torch.cuda.ExternalStream(b.stream)
            torch.cuda.synchronize()
    elif kind == "roundtrip":
        st["host"] = [torch.from_numpy(a).pin_memory() for a in sim.download()]
        st["back"] = [torch.empty_like(a).pin_memory() for a in st["host"][1:]]
    elif kind == "rollout":
        mass, pos, vel = sim.download()
        rng = np.random.default_rng(seed)
        drift = pos + (case["dt"] * case["steps"]) * vel
        target = drift + 1e-3 * rng.standard_normal(pos.shape)
        st.update(mass=mass, pos=pos, vel=vel, target=target.astype(np.float32),
                  steps=case["steps"], every=case["every"])
    elif kind == "render":
        r = bh.Renderer(sim, case["width"], case["height"])
        r.zoomCamera(case["zoom"], case["width"] / 2, case["height"] / 2)
        density, image = r.targets()
        shape = (case["height"], case["width"])
        st["renderer"] = r
        owner = (r, sim)
        st["out"] = {"density": _view(owner, density, shape),
                     "image": _view(owner, image, shape + (4,), "|u1")}
    return st


def run(state):
    sim, kind = state["sim"], state["kind"]
    if kind == "step":
        sim.getCommands().submit()
        return state["out"]
    if kind == "restart":
        with torch.cuda.stream(state["stream"]):
            for name, value in state["start"].items():
                state["out"][name].copy_(value)
        sim.getCommands().submit()
        return state["out"]
    if kind == "roundtrip":
        sim.upload(*state["host"])
        sim.step(1)
        pos, vel = state["back"]
        sim.download_into(None, pos, vel)
        return {"pos": pos, "vel": vel}
    if kind == "forces":
        return sim.computeAccelerations()
    if kind == "rollout":
        sim.upload(state["mass"], state["pos"], state["vel"])
        loss, gx, gv, gm = sim.rollout_grad(state["steps"], state["every"], state["target"])
        return {"loss": loss, "pos": gx, "vel": gv, "mass": gm}
    if kind == "render":
        state["renderer"].getCommands().submit()
        return state["out"]
    return sim.diagnostics()


def work(case):
    if case["kind"] == "render":
        # positions and radii in, density and image out; a few flops a pixel of each disc
        px = case["width"] * case["height"]
        return {"bytes": 12.0 * case["n"] + 8.0 * px, "flops": 150.0 * case["n"] + 20.0 * px}
    if "systems" in case:
        n = case["systems"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        size = n / case["systems"]
    else:
        n = size = float(case["n"])
    if case["kind"] == "diagnose":
        return {"bytes": 20.0 * n, "flops": 10.0 * n * (n - 1) / 2}
    # Tree code: about 4 log2(n) / theta^2 interactions a body (307 a body were
    # counted at 800k bodies and theta 0.5), 16 flops each at least.
    flops = 16.0 * n * 4.0 * math.log2(size) / case["theta"] ** 2
    if case["kind"] == "forces":
        return {"bytes": 20.0 * n, "flops": flops}
    if case["kind"] == "rollout":
        # forward steps and as many backward ones (about twice a force each)
        return {"bytes": (20.0 + 8.0 + 20.0) * n, "flops": 3.0 * flops * case["steps"]}
    kdk = case["integrator"] == "leapfrog-kdk"
    return {"bytes": (20.0 + 16.0 + (16.0 if kdk else 0.0)) * n, "flops": flops}


# ---- the same results in FP64, by direct sums ---------------------------------

_PAIRS = 1 << 26  # pairs held at a time
_MAX_DIRECT = 400_000


def _soft2(case, mi, mj):
    """Squared softening of each pair: constant, or the reference's G dt max(m_i, m_j)."""
    if case["softening"] == "plummer":
        return float(np.float32(case["eps"])) ** 2
    return float(np.float32(case["dt"])) * torch.maximum(mi[:, None], mj[None, :])


def _rows(n):
    step = max(1, _PAIRS // n)
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _forces(case, x, m):
    """a_i = sum_j m_j (x_j - x_i) / (|x_j - x_i|^2 + eps_ij^2)^(3/2), G = 1."""
    n = x.shape[0]
    out = torch.empty_like(x)
    for a, b in _rows(n):
        dx = x[None, :, 0] - x[a:b, None, 0]
        dy = x[None, :, 1] - x[a:b, None, 1]
        w = (dx * dx).addcmul_(dy, dy).add_(_soft2(case, m[a:b], m))
        w = w.pow_(-1.5).mul_(m[None, :])
        w = torch.where(torch.isfinite(w), w, torch.zeros_like(w))
        out[a:b, 0] = (w * dx).sum(1)
        out[a:b, 1] = (w * dy).sum(1)
    return out


def _force_vjp(case, x, m, abar):
    """(da/dx)^T abar and (da/dm)^T abar of the direct sum with constant softening."""
    n = x.shape[0]
    e2 = _soft2(case, m, m)
    xbar, mbar = torch.zeros_like(x), torch.zeros_like(m)
    for a, b in _rows(n):
        dx = x[None, :, 0] - x[a:b, None, 0]
        dy = x[None, :, 1] - x[a:b, None, 1]
        s2 = 1.0 / (dx * dx + dy * dy + e2)
        s3 = s2 * s2.sqrt()
        ax, ay = abar[a:b, None, 0], abar[a:b, None, 1]
        ar = ax * dx + ay * dy
        mbar += (ar * s3).sum(0)
        t = -3.0 * s3 * s2 * ar
        rx = m[None, :] * (s3 * ax + t * dx)
        ry = m[None, :] * (s3 * ay + t * dy)
        xbar[:, 0] += rx.sum(0)
        xbar[:, 1] += ry.sum(0)
        xbar[a:b, 0] -= rx.sum(1)
        xbar[a:b, 1] -= ry.sum(1)
    return xbar, mbar


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


def exact(case, seed):
    sim = _simulation(case, seed)
    n = sim.getNumBodies()
    kind = case["kind"]
    if n > _MAX_DIRECT and kind not in ("render",) and "systems" not in case:
        return None
    mass, pos, vel = (_f64(a) for a in sim.download())
    dt = float(np.float32(case["dt"]))
    if kind == "forces":
        # walks of monopoles only are 10% off the direct sum at these thetas
        monopole = case["walk"] == "exact" or case["multipole"] == 1
        return None if monopole else _forces(case, pos, mass)
    if kind in ("step", "restart", "roundtrip"):
        offsets = [int(o) for o in sim.offsets] if "systems" in case else [0, n]

        def force(x):
            return torch.cat([_forces(case, x[a:b], mass[a:b])
                              for a, b in zip(offsets, offsets[1:])])
        if case["integrator"] == "leapfrog-kdk":
            v = vel + 0.5 * dt * force(pos)
            x = pos + dt * v
            acc = force(x)
            return {"pos": x, "vel": v + 0.5 * dt * acc,
                    "acc": None if case["multipole"] == 1 else acc}
        v = vel + dt * force(pos)
        if kind == "restart":
            # the per-body monopole walk at these settings is 10% off the direct
            # sum, and the kick is larger than the initial velocities
            return {"pos": pos + dt * v, "vel": None}
        return {"pos": pos + dt * v, "vel": v}
    if kind == "rollout":
        target = _f64(prepare(case, seed)["target"])
        xs, v, a = [pos], vel, _forces(case, pos, mass)
        for _ in range(case["steps"]):
            v = v + 0.5 * dt * a
            xs.append(xs[-1] + dt * v)
            a = _forces(case, xs[-1], mass)
            v = v + 0.5 * dt * a
        miss = xs[-1] - target
        xbar, vbar = 2.0 / n * miss, torch.zeros_like(vel)
        mbar, pending = torch.zeros_like(mass), torch.zeros_like(vel)
        for x in reversed(xs[1:]):
            dx, dm = _force_vjp(case, x, mass, pending + 0.5 * dt * vbar)
            xbar, mbar = xbar + dx, mbar + dm
            vbar = vbar + dt * xbar
            pending = 0.5 * dt * vbar
        dx, dm = _force_vjp(case, xs[0], mass, pending)
        return {"loss": miss.square().sum() / n, "pos": xbar + dx, "vel": vbar, "mass": mbar + dm}
    if kind == "render":
        return {"density": _density(case, sim, pos, n), "image": None}
    return _conserved(case, mass, pos, vel)


def _density(case, sim, pos, n):
    """The density pass: exp(-10 r^2) discs of radius 2 radiusMultiplier pixels."""
    radius = _f64(sim.read_buffer("radius_multiplier", np.float32, n))
    w, h = case["width"], case["height"]
    hy = 10.0 * case["zoom"]
    hx = hy * w / h
    centre = torch.stack([(pos[:, 0] / hx + 1.0) * 0.5 * w, (pos[:, 1] / hy + 1.0) * 0.5 * h], 1)
    weight = torch.where(radius > 1.0, 0.1, 0.02).double() / (1.0 + 0.05 * max(hx, hy))
    out = torch.zeros(h * w, dtype=torch.float64, device="cuda")
    for mult in torch.unique(radius).tolist():
        at = radius == mult
        c, wt, R = centre[at], weight[at], 2.0 * mult
        first = torch.ceil(c - R - 0.5)
        reach = int(math.floor(2.0 * R)) + 2
        for j in range(reach):
            for i in range(reach):
                px, py = first[:, 0] + i, first[:, 1] + j
                r2 = ((px + 0.5 - c[:, 0]).square() + (py + 0.5 - c[:, 1]).square()) / (R * R)
                ok = (r2 <= 1.0) & (px >= 0) & (px < w) & (py >= 0) & (py < h)
                cell = (py[ok] * w + px[ok]).long()
                out.index_add_(0, cell, wt[ok] * torch.exp(-10.0 * r2[ok]))
    return out.reshape(h, w)


def _conserved(case, m, x, v):
    n = x.shape[0]
    pair = torch.zeros((), dtype=torch.float64, device="cuda")
    for a, b in _rows(n):
        dx = x[None, :, 0] - x[a:b, None, 0]
        dy = x[None, :, 1] - x[a:b, None, 1]
        w = (dx * dx).addcmul_(dy, dy).add_(_soft2(case, m[a:b], m)).rsqrt_()
        w[torch.arange(b - a, device="cuda"), torch.arange(a, b, device="cuda")] = 0.0
        pair += (m[a:b] * (w @ m)).sum()
    kinetic = float(0.5 * (m * v.square().sum(1)).sum())
    potential = float(-0.5 * pair)
    total = float(m.sum())
    com = [float(c) for c in (m[:, None] * x).sum(0) / total]
    return {"total_mass": total, "com": com, "momentum": [float(c) for c in (m[:, None] * v).sum(0)],
            "angular_momentum": float((m * (x[:, 0] * v[:, 1] - x[:, 1] * v[:, 0])).sum()),
            "kinetic_energy": kinetic, "potential_energy": potential,
            "total_energy": kinetic + potential}
