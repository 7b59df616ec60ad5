"""The work that this framework is timed on: what its users have it do, through
its public entry points, over the sizes and options that they use.

Six kinds of call:

* ``run``      a simulation in its steady state advanced by some steps, then its state read back, as a
               program does between two dumps (Engine.run, Engine.download_fields, Engine.energy)
* ``fresh``    a new start configuration: upload, list build, the first steps from random positions, read back
* ``ensemble`` many independent sphere systems in one engine (ensemble.sphere_ensemble), advanced and read back
* ``fire``     many quenched packings in the slow approach to their minima, some FIRE iterations
               (ensemble.plane_fire_ensemble, Engine.minimize)
* ``network``  the learned warm start: a training step, or the prediction alone (warmstart.WarmStartNet)
* ``forces``   one evaluation of forces and torques from a caller's device arrays (sg_compute_static)

The programs (potential, aligner, integrator, constraint, parameters, densities)
are those of this repository's benchmark and configurations.
"""
import ctypes

import numpy as np
import torch

from samos_b200 import Engine, Simulation, engine
from samos_b200.ensemble import SphereReplica, plane_fire_ensemble, sphere_ensemble
from samos_b200.warmstart import WarmStartNet

_RADII = {"k": "10", "use_particle_radii": ""}
_LJ = {"epsilon": "1", "sigma": "1", "rcut": "2.5", "shifted": ""}
_ABP = ("brownian", {"v0": "0.5", "nu": "0.1", "mu": "1", "mur": "1", "seed": "3"})
_PLANE = ("x", "y", "nx", "ny", "vx", "vy")
_SPACE = ("x", "y", "z", "nx", "ny", "nz", "vx", "vy", "vz")

#: program -> start geometry, pair potential, aligner, integrator, time step, fields read back, and the bytes of a
#: particle's state that a step reads and writes (plane: x y nx ny r in, x y nx ny vx vy out; space: with z too)
PROGRAMS = {
    "disks_nematic": ("bidisperse", ("soft", _RADII), ("nematic", {"J": "0.5"}),
                      ("brownian", {"v0": "0.3", "nu": "0.1", "mu": "1", "mur": "1", "seed": "1"}), 5e-4, _PLANE, 88),
    "disks_polar": ("polydisperse", ("soft", _RADII), ("polar", {"J": "0.1"}),
                    ("brownian", {"v0": "0.5", "nu": "0.1", "mu": "1", "mur": "1", "seed": "2"}), 1e-3, _PLANE, 88),
    "sphere_polar": ("sphere", ("soft", _RADII), ("polar", {"J": "0.2"}),
                     ("brownian", {"v0": "1.0", "nu": "0.05", "mu": "1", "mur": "1", "seed": "3"}), 1e-3, _SPACE, 128),
    "torus_polar": ("torus", ("soft", {"k": "10"}), ("polar", {"J": "0.2"}),
                    ("brownian", {"v0": "1.0", "nu": "0.05", "mu": "1", "mur": "1", "seed": "3"}), 1e-3, _SPACE, 128),
    "lj_polar": ("lattice", ("lj", _LJ), ("polar", {"J": "0.2"}), _ABP, 1e-4, _PLANE, 88),
    "morse_polar": ("lattice", ("morse", {"D": "1", "a": "2", "re": "2", "rcut": "2.5", "shifted": ""}),
                    ("polar", {"J": "0.2"}), _ABP, 1e-3, _PLANE, 88),
    "gaussian_polar": ("lattice", ("gaussian", {"A": "2", "B": "-1", "alpha": "1", "beta": "3", "rA": "0", "rB": "1.5",
                                                "rcut": "2.5"}), ("polar", {"J": "0.2"}), _ABP, 1e-3, _PLANE, 88),
    "vicsek": ("lattice", ("soft", {"k": "10"}), ("vicsek", {"rcut": "2.0"}),
               ("vicsek", {"v0": "0.5", "eta": "0.3", "mu": "0.1", "seed": "5"}), 1e-2, _PLANE, 88),
    "lj_langevin": ("lattice", ("lj", _LJ), None,
                    ("langevin", {"gamma": "1", "seed": "7", "method": "baoab", "min_val": "0.5"}), 1e-4, _PLANE, 88),
    "nve_polar": ("lattice", ("soft", {"k": "1"}), ("polar", {"J": "1"}), ("nve", {"limit": "0.0001"}), 1e-3, _PLANE, 88),
}
#: steps before a steady-state case is handed over: overlaps relaxed, the engine's kernels chosen
WARM = 400


def listed():
    return [
        # the smallest configuration, between two log lines: 16 blocks, so latency and launches count
        {"name": "disks_2k", "kind": "run", "program": "disks_polar", "n": 2000, "steps": 100},
        # the sphere configuration
        {"name": "sphere_64k", "kind": "run", "program": "sphere_polar", "n": 65536, "steps": 60},
        # the headline configuration
        {"name": "disks_4M", "kind": "run", "program": "disks_nematic", "n": 4194304, "steps": 60},
        # passive liquids: thermostatted and at constant energy, odd sizes
        {"name": "lj_langevin_250k", "kind": "run", "program": "lj_langevin", "n": 250007, "steps": 60},
        {"name": "nve_20k", "kind": "run", "program": "nve_polar", "n": 20011, "steps": 100},
        # another pair potential, the Vicsek model, and a curved surface with an iterative projection
        {"name": "morse_500k", "kind": "run", "program": "morse_polar", "n": 500009, "steps": 40},
        {"name": "vicsek_130k", "kind": "run", "program": "vicsek", "n": 131101, "steps": 60},
        {"name": "torus_50k", "kind": "run", "program": "torus_polar", "n": 50021, "steps": 60},
        # 256 replicas of uneven size, as in a parameter scan
        {"name": "ensemble_256", "kind": "ensemble", "replicas": 256, "n_lo": 1024, "n_hi": 65536, "steps": 60},
        # relaxing packings: where nearly all of a minimisation's iterations are spent
        {"name": "fire_32", "kind": "fire", "replicas": 32, "n_lo": 1024, "n_hi": 16384, "steps": 250},
        # one optimiser step of the warm-start network on a batch of packings
        {"name": "train_64", "kind": "network", "replicas": 64, "n": 4096, "train": True},
        # one force evaluation of a middle-sized system from device arrays
        {"name": "forces_30k", "kind": "forces", "n": 30011, "align": "nematic", "radii": True},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["run"] * 8 + ["fresh", "ensemble", "fire", "fire", "network", "network", "forces", "forces"])
    if kind == "run":
        program = rng.choice(sorted(PROGRAMS) + ["disks_nematic", "disks_polar", "sphere_polar"])
        n = _log(rng, 500, 1500000 if program in ("disks_nematic", "disks_polar", "sphere_polar") else 400000)
        return {"kind": kind, "program": program, "n": n, "steps": max(10, min(_log(rng, 20, 200), 40000000 // n))}
    if kind == "fresh":
        return {"kind": kind, "program": rng.choice(["disks_nematic", "disks_polar", "sphere_polar"]),
                "n": _log(rng, 10000, 1000000), "steps": 20}
    if kind == "ensemble":
        return {"kind": kind, "replicas": _log(rng, 2, 200), "n_lo": _log(rng, 300, 2000), "n_hi": _log(rng, 2500, 40000),
                "steps": rng.randint(20, 60)}
    if kind == "fire":
        return {"kind": kind, "replicas": _log(rng, 1, 48), "n_lo": _log(rng, 256, 2000), "n_hi": _log(rng, 2100, 12000),
                "steps": rng.randint(100, 300)}
    if kind == "network":
        return {"kind": kind, "replicas": _log(rng, 1, 60), "n": 2 * _log(rng, 256, 2500), "train": rng.random() < 0.5}
    return {"kind": kind, "n": _log(rng, 200, 65536), "align": rng.choice(["nematic", "polar", "none"]),
            "radii": rng.random() < 0.7}


# -- inputs ----------------------------------------------------------------------------------------------------
def _disks(n, phi, radius, rng):
    """n disks uniform in a square periodic box of packing fraction phi (overlaps allowed), random directors."""
    L = float(np.sqrt(np.sum(np.pi * radius * radius) / phi))
    th = rng.uniform(0.0, 2.0 * np.pi, n)
    zero = np.zeros(n)
    return dict(x=rng.uniform(-L / 2, L / 2, n), y=rng.uniform(-L / 2, L / 2, n), z=zero, vx=zero, vy=zero, vz=zero,
                nx=np.cos(th), ny=np.sin(th), nz=zero, radius=radius), L


def _bidisperse(n, rng):
    r = np.where(np.arange(n) % 2 == 0, 1.0, 1.4)
    rng.shuffle(r)
    return r


def _lattice(n, phi, rng):
    """Unit disks on a square lattice, jittered by up to 0.1: no overlaps, so steep potentials start finite."""
    m, a = int(np.ceil(np.sqrt(n))), float(np.sqrt(np.pi / phi))
    L, k, zero, th = m * a, np.arange(n), np.zeros(n), rng.uniform(0.0, 2.0 * np.pi, n)
    return dict(x=-L / 2 + (k % m + 0.5) * a + rng.uniform(-0.1, 0.1, n),
                y=-L / 2 + (k // m + 0.5) * a + rng.uniform(-0.1, 0.1, n), z=zero, vx=zero, vy=zero, vz=zero,
                nx=np.cos(th), ny=np.sin(th), nz=zero, radius=np.ones(n)), L


def _sphere(n, rng):
    """Unit particles uniform on the sphere that they cover once, random tangent directors."""
    R = float(np.sqrt(n / 4.0))
    z, ph = rng.uniform(-R, R, n), rng.uniform(0.0, 2.0 * np.pi, n)
    s = np.sqrt(np.maximum(R * R - z * z, 0.0))
    pos = np.stack([s * np.cos(ph), s * np.sin(ph), z])
    t = rng.standard_normal((3, n))
    t -= np.sum(t * pos, 0) / (R * R) * pos
    t /= np.linalg.norm(t, axis=0)
    zero = np.zeros(n)
    return dict(x=pos[0], y=pos[1], z=pos[2], vx=zero, vy=zero, vz=zero, nx=t[0], ny=t[1], nz=t[2],
                radius=np.ones(n)), R


def _torus(n, rng):
    """Unit particles on a torus of tube radius a = c/3 at packing fraction 0.5."""
    c = float(np.sqrt(3.0 * n / (2.0 * np.pi)))
    a = c / 3.0
    u, v = rng.uniform(0.0, 2.0 * np.pi, n), rng.uniform(0.0, 2.0 * np.pi, n)
    zero = np.zeros(n)
    return dict(x=(c + a * np.cos(v)) * np.cos(u), y=(c + a * np.cos(v)) * np.sin(u), z=a * np.sin(v), vx=zero, vy=zero,
                vz=zero, nx=-np.sin(u), ny=np.cos(u), nz=zero, radius=np.ones(n)), c, a


def _start(case, seed):
    """(particles, box sides, periodic, constraint, neighbour list) of a run or fresh case."""
    geometry, n, rng = PROGRAMS[case["program"]][0], case["n"], np.random.default_rng(seed)
    if geometry == "sphere":
        parts, R = _sphere(n, rng)
        return parts, (2 * R + 6.0,) * 3, False, ("sphere", {"r": repr(R)}), (2.4, 0.3)
    if geometry == "torus":
        parts, c, a = _torus(n, rng)
        side = 2 * (c + a) + 20
        return parts, (side, side, 2 * a + 20), False, ("torus", {"c": repr(c), "a": repr(a)}), (2.4, 0.3)
    if geometry == "polydisperse":
        parts, L = _disks(n, 0.6, rng.uniform(0.9, 1.1, n), rng)
        rc = 2.4
    elif geometry == "bidisperse":
        parts, L = _disks(n, 0.8, _bidisperse(n, rng), rng)
        rc = 2.8
    else:
        parts, L = _lattice(n, 0.6, rng)
        rc = 2.8
    return parts, (L, L, 10.0), True, ("plane", {}), (rc, 0.3)


def _simulation(case, seed):
    _, pair, align, integrator, dt, _, _ = PROGRAMS[case["program"]]
    parts, box, periodic, constraint, nlist = _start(case, seed)
    sim = Simulation(Engine(case["n"]))
    sim.box(*box, periodic)
    sim.b.upload_fields(parts)
    sim.nlist(*nlist)
    sim.constraint(*constraint)
    sim.pair_potential(*pair)
    if align:
        sim.pair_align(*align)
    sim.timestep(dt)
    sim.integrator(*integrator)
    sim.commit()
    return sim, parts


def _spread(case):
    """Replica sizes, evenly log-uniform over the case's range and in no order; the same for every seed."""
    lo, hi, count = case["n_lo"], case["n_hi"], case["replicas"]
    sizes = lo * (hi / lo) ** ((np.arange(count) + 0.5) / count)
    return [int(round(v)) for v in np.random.default_rng(count).permutation(sizes)]


def _packings(sizes, rng):
    return [_disks(n, rng.uniform(0.84, 0.90), _bidisperse(n, rng), rng) for n in sizes]


def _targets(case, rng):
    return [rng.normal(0.0, 0.3, (case["n"], 2)) for _ in range(case["replicas"])]


def _weights(rng):
    """The network's parameters, uniform by fan-in (layer inputs 4, 4, 64, 64, 64, 64, 4, 64), the output ones small."""
    sizes = ((256, 4), (64, 4), (4096, 64), (64, 64), (8192, 64), (64, 64), (256, 4), (64, 6400), (1, 64))
    return np.concatenate([rng.uniform(-1.0, 1.0, size) / np.sqrt(fan_in) for size, fan_in in sizes]).astype(np.float32)


#: a learning rate, and optimiser moments as in the middle of a training
_LR, _STEP, _MOMENT2 = 1e-3, 1000, 1e-4


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "fresh"):
        sim, parts = _simulation(case, seed)
        fields = PROGRAMS[case["program"]][5]
        state = dict(case=case, sim=sim, fields=fields, out={f: engine.pinned_empty(case["n"]) for f in fields})
        sim.run(WARM - 1)
        if kind == "fresh":
            state["parts"] = {f: engine.pinned_copy(v) for f, v in parts.items()}
        return state
    rng = np.random.default_rng(seed)
    if kind == "ensemble":
        reps = []
        for n in _spread(case):
            parts, R = _sphere(n, rng)
            reps.append(SphereReplica(parts=parts, R=R, v0=rng.uniform(0.01, 1.0), J=rng.uniform(0.0, 1.0),
                                      nu=float(np.exp(rng.uniform(np.log(1e-3), 0.0))), seed=int(rng.integers(1, 2**31 - 1))))
        eng = sphere_ensemble(reps)
        eng.run(WARM // 2 - 1)
        return dict(case=case, eng=eng, out={f: engine.pinned_empty(sum(eng.n)) for f in _SPACE})
    if kind == "fire":
        insts = _packings(_spread(case), rng)
        eng = plane_fire_ensemble(insts)
        eng.build_nlist()
        eng.minimize(1500)
        start = []
        for r, n in enumerate(eng.n):
            flat = {f: engine.pinned_empty(n) for f in ("x", "y", "vx", "vy")}
            eng.download_fields(("x", "y"), replica=r, out=flat)
            flat["vx"][:] = flat["vy"][:] = 0.0
            start.append(flat)
        return dict(case=case, eng=eng, start=start, out={f: engine.pinned_empty(sum(eng.n)) for f in ("x", "y", "fx", "fy")})
    if kind == "network":
        insts = _packings([case["n"]] * case["replicas"], rng)
        eng = plane_fire_ensemble(insts)
        net = WarmStartNet()
        net.set_params(_weights(rng))
        net.m.zero_()
        net.v.fill_(_MOMENT2)
        net.step = _STEP
        ids = net.slot_ids(eng)
        slot_of = np.empty(sum(eng.n), np.int64)  # particle, over all replicas -> slot
        at = 0
        for r, n in enumerate(eng.n):
            off = eng.replica_slots(r)[0]
            slot_of[at + ids[off:off + n]] = np.arange(off, off + n)
            at += n
        return dict(case=case, eng=eng, net=net, box=net.box_array(eng), n=at, slot_of=torch.from_numpy(slot_of).cuda(),
                    target=net.slot_targets(eng, _targets(case, rng)))
    parts, L = _disks(case["n"], 0.8, _bidisperse(case["n"], rng), rng)
    ins = [torch.from_numpy(parts[f]).cuda() for f in ("x", "y", "z", "nx", "ny", "nz", "radius")]
    outs = {f: torch.empty(case["n"], dtype=torch.float64, device="cuda") for f in ("fx", "fy", "fz", "tx", "ty", "tz")}
    return dict(case=case, lib=engine.load(), L=L, ins=ins, outs=outs)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("run", "fresh"):
        eng = state["sim"].b
        if kind == "fresh":
            eng.upload_fields(state["parts"])
            eng.build_nlist()
        eng.run(case["steps"] - 1)  # `run N` performs N + 1 steps
        out = dict(eng.download_fields(state["fields"], out=state["out"]))
        out["energy"] = eng.energy(0, 0)
        return out
    if kind == "ensemble":
        eng, out, at = state["eng"], state["out"], 0
        eng.run(case["steps"] - 1)
        for r, n in enumerate(eng.n):
            eng.download_fields(_SPACE, replica=r, out={f: out[f][at:at + n] for f in _SPACE})
            at += n
        return dict(out)
    if kind == "fire":
        eng, out, at = state["eng"], state["out"], 0
        for r, flat in enumerate(state["start"]):
            eng.upload_fields(flat, replica=r)
            eng.set_replica_param(r, 4, 0, 0, 0.01)  # FIRE's time step and mixing start over
            eng.set_replica_param(r, 4, 0, 1, 0.1)
        eng.positions_changed()
        eng.minimize(case["steps"] - 1)
        for r, n in enumerate(eng.n):
            eng.download_fields(("x", "y", "fx", "fy"), replica=r, out={f: out[f][at:at + n] for f in out})
            at += n
        return dict(out, energy=[eng.energy(0, 0, r) for r in range(len(eng.n))])
    if kind == "network":
        net = state["net"]
        if not case["train"]:
            return net.forward(state["eng"], state["box"]).view(-1, 2)[state["slot_of"]]
        loss = net.loss_and_grad(state["eng"], state["box"], state["target"], state["n"])
        net.adam_step(_LR)
        return dict(loss=loss, grad=net.grad, params=net.params)
    p, L, outs = (lambda t: ctypes.c_void_p(t.data_ptr())), state["L"], state["outs"]
    rc = state["lib"].sg_compute_static(
        case["n"], L, L, 10.0, 1, 2.8, 0.3, *map(p, state["ins"]), 10.0, 2.0, int(case["radii"]),
        engine.ALIGN.get(case["align"], -1), 0.5, 2.8, *map(p, outs.values()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError("sg_compute_static: %d" % rc)
    return dict(outs)


def work(case):
    """Bytes: the state that every step reads and writes, and what goes to and from the host. Operations: about 30 for a
    neighbour pair and 200 for a particle's own update; the network's products and edge passes."""
    kind = case["kind"]
    if kind in ("run", "fresh"):
        per, fields = PROGRAMS[case["program"]][6], len(PROGRAMS[case["program"]][5])
        n, pairs = case["n"], 5.2
        moved = 8 * fields + (80 if kind == "fresh" else 0)
        return {"bytes": n * (case["steps"] * per + moved), "flops": n * case["steps"] * (200 + 30 * pairs)}
    if kind in ("ensemble", "fire"):
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["replicas"] * (hi - lo) / np.log(hi / lo)  # the mean of a log-uniform size
        per, moved = (128, 72) if kind == "ensemble" else (88, 64)
        return {"bytes": n * (case["steps"] * per + moved), "flops": n * case["steps"] * (200 + 30 * 6)}
    if kind == "network":
        n, passes = case["n"] * case["replicas"], 3 if case["train"] else 1
        # positions, radius, list entries in; displacement out; two 64-wide layers and the edges around them
        return {"bytes": n * (24 + 4 * 7 + 8 + (16 if case["train"] else 0)) * 1.0,
                "flops": passes * n * (2.0 * 64 * 192 + 7 * 64 * 22.0)}
    return {"bytes": case["n"] * 13 * 8.0, "flops": case["n"] * 4.5 * 40.0}


# -- what the outputs are in 64 bits ----------------------------------------------------------------------------
def _wrap(d, L):
    return torch.where(d > L / 2, d - L, torch.where(d < -L / 2, d + L, d))


def _soft_and_align(pos, dirs, contact, k, J, rc, L, nematic, rows):
    """Forces and torques over all pairs of the particles in `rows` with everybody: soft repulsion, and J n_i x n_j."""
    d = pos[None, :, :] - pos[rows, None, :]
    if L is not None:
        d = _wrap(d, L)
    r = d.square().sum(-1).sqrt()
    sig = contact[rows, None] + contact[None, :]
    other = torch.ones_like(r, dtype=torch.bool)
    other[torch.arange(len(rows), device=r.device), rows] = False
    ff = torch.where(other & (r < sig), k * (sig - r) / r.clamp_min(1e-300), 0.0)
    force = -(ff[..., None] * d).sum(1)
    w = (other & (r <= rc)).to(r.dtype) * J
    if nematic:
        w = w * (dirs[rows] @ dirs.T)
    return force, torch.cross(dirs[rows], w @ dirs, dim=1)


def _gauss(seed, counter):
    """The documented noise stream: Philox-4x32-10 on (counter, 0, 0) under (seed, 0x53414D4F), then Box-Muller."""
    m = np.uint64(0xFFFFFFFF)
    c = [counter & m, counter >> np.uint64(32), np.zeros_like(counter), np.zeros_like(counter)]
    k0, k1 = seed, 0x53414D4F
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((p >> np.uint64(5)).astype(float) * 67108864.0 + (q >> np.uint64(6)).astype(float)) / 9007199254740992.0
         for p, q in ((c[0], c[1]), (c[2], c[3]))]
    return np.sqrt(-2.0 * np.log(u[0] + 1.0 / 9007199254740992.0)) * np.cos(2.0 * np.pi * u[1])


def _exact_run(case, seed, dev):
    _, _, (align, ap), (_, ip), dt, fields, _ = PROGRAMS[case["program"]]
    parts, box, periodic, constraint, nlist = _start(case, seed)
    n, steps = case["n"], case["steps"] + (WARM if case["kind"] == "run" else 0)
    t = {f: torch.from_numpy(v).to(dev) for f, v in parts.items()}
    pos, dirs = torch.stack([t["x"], t["y"], t["z"]], 1), torch.stack([t["nx"], t["ny"], t["nz"]], 1)
    v0, nu, noise_seed = float(ip["v0"]), float(ip["nu"]), int(ip["seed"])
    J = float(ap["J"]) * (2.0 if align == "nematic" else 1.0)
    L, R = (box[0], None) if periodic else (None, float(constraint[1]["r"]))
    rows, up = torch.arange(n, device=dev), torch.tensor([0.0, 0.0, 1.0], device=dev, dtype=torch.float64)
    for s in range(steps):
        force, torque = _soft_and_align(pos, dirs, t["radius"], 10.0, J, nlist[0], L, align == "nematic", rows)
        vel = v0 * dirs + force
        pos = pos + dt * vel
        if L is not None:
            pos, normal = torch.stack([_wrap(pos[:, 0], L), _wrap(pos[:, 1], L), pos[:, 2]], 1), up.expand(n, 3)
        else:
            pos = pos * (R / pos.norm(dim=1, keepdim=True))
            normal = pos / R
            vel = vel - (vel * normal).sum(1, keepdim=True) * normal
            dirs = dirs - (dirs * normal).sum(1, keepdim=True) * normal
            dirs = dirs / dirs.norm(dim=1, keepdim=True)
        turn = dt * (torque * normal).sum(1) + np.sqrt(nu * dt) * torch.from_numpy(
            _gauss(noise_seed, np.uint64(s) * np.uint64(n) + np.arange(n, dtype=np.uint64))).to(dev)
        dirs = dirs * turn.cos()[:, None] + torch.cross(normal, dirs, dim=1) * turn.sin()[:, None]
        dirs = dirs / dirs.norm(dim=1, keepdim=True)
    flat = dict(x=pos[:, 0], y=pos[:, 1], z=pos[:, 2], nx=dirs[:, 0], ny=dirs[:, 1], nz=dirs[:, 2], vx=vel[:, 0],
                vy=vel[:, 1], vz=vel[:, 2])
    return dict({f: flat[f].cpu().numpy() for f in fields}, energy=None)


def _exact_network(case, seed, dev):
    rng = np.random.default_rng(seed)
    insts = _packings([case["n"]] * case["replicas"], rng)
    P = torch.from_numpy(_weights(rng).astype(np.float64)).to(dev).requires_grad_(case["train"])
    targets = _targets(case, rng)
    W1a, b1a, W1b, b1b = P[:256].view(64, 4), P[256:320], P[320:4416].view(64, 64), P[4416:4480]
    Wpq, b2, W2e, w2, c = P[4480:12672].view(64, 128), P[12672:12736], P[12736:12992].view(64, 4), P[12992:13056], P[13056]
    grad, loss, disps, total = torch.zeros_like(P), 0.0, [], case["n"] * case["replicas"]
    for (parts, L), target in zip(insts, targets):
        pos = torch.from_numpy(np.stack([parts["x"], parts["y"]], 1)).to(dev)
        rad = torch.from_numpy(parts["radius"]).to(dev)
        found = [torch.cat([((_wrap(pos[None] - pos[a:a + 2048, None], L).square().sum(-1) < 2.8 * 2.8).nonzero()
                             + torch.tensor([a, 0], device=dev)) for a in range(0, len(pos), 2048)])]
        i, j = found[0].T
        i, j = i[i != j], j[i != j]
        d = _wrap(pos[j] - pos[i], L)
        r = d.norm(dim=1)
        e = torch.stack([r, rad[i], rad[j], rad[i] + rad[j] - r], 1)
        s = torch.zeros(len(pos), 64, dtype=torch.float64, device=dev).index_add(0, i, torch.relu(e @ W1a.T + b1a))
        PQ = torch.relu(s @ W1b + b1b) @ Wpq
        w = torch.relu(PQ[i, :64] + PQ[j, 64:] + e @ W2e.T + b2) @ w2 + c
        disp = torch.zeros_like(pos).index_add(0, i, w[:, None] * d / r[:, None])
        if case["train"]:
            part = (disp - torch.from_numpy(target).to(dev)).square().sum() / total
            grad += torch.autograd.grad(part, P)[0]
            loss += float(part)
        disps.append(disp.detach())
    if not case["train"]:
        return torch.cat(disps)
    step, m, v = _STEP + 1, 0.1 * grad, 0.999 * _MOMENT2 + 0.001 * grad * grad
    params = P.detach() - _LR * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return dict(loss=loss, grad=grad, params=params)


def exact(case, seed):
    """None for the trajectories that all pairs in 64 bits would take too long for, for those of the other programs, and for
    FIRE, whose path follows the order of its own sums."""
    dev, kind = "cuda" if torch.cuda.is_available() else "cpu", case["kind"]
    if kind in ("run", "fresh"):
        small = case["n"] <= 4096 and case["program"] in ("disks_nematic", "disks_polar", "sphere_polar")
        return _exact_run(case, seed, dev) if small and kind == "run" else None
    if kind == "network":
        return _exact_network(case, seed, dev)
    if kind != "forces":
        return None
    rng = np.random.default_rng(seed)
    n = case["n"]
    parts, L = _disks(n, 0.8, _bidisperse(n, rng), rng)
    t = {f: torch.from_numpy(v).to(dev) for f, v in parts.items()}
    pos, dirs = torch.stack([t["x"], t["y"], t["z"]], 1), torch.stack([t["nx"], t["ny"], t["nz"]], 1)
    contact = t["radius"] if case["radii"] else torch.ones_like(t["radius"])  # the default contact distance a = 2
    J = {"nematic": 1.0, "polar": 0.5, "none": 0.0}[case["align"]]
    got = [_soft_and_align(pos, dirs, contact, 10.0, J, 2.8, L, case["align"] == "nematic", rows)
           for rows in torch.arange(n, device=dev).split(1024)]
    force, torque = (torch.cat(v) for v in zip(*got))
    return dict(fx=force[:, 0], fy=force[:, 1], fz=force[:, 2], tx=torque[:, 0], ty=torque[:, 1], tz=torque[:, 2])
