"""The engine's measured workloads: what a program that evolves self-gravitating
discs has this framework do, from one small galaxy to millions of bodies.

Every case goes through the public entry points (``galaxy_b200.nbody_gpu``,
``galaxy_b200.batch``, ``galaxy_b200.serve``).  Sizes, opening angles, leaf
sizes, softenings and time steps are those of the benchmark's configurations,
the receipt tool and the tests, with odd sizes among them.  Kinds of case:

* ``evolve``    resident simulation: fused KDK steps, then a snapshot of the state
* ``solve``     tree rebuild + force on a given state, accelerations read back,
                FP64 invariants (the boundary solve and the diagnostics cadence)
* ``loop``      the reference host's own loop: kick_drift, rebuild, force,
                final_kick called one by one, then a snapshot
* ``batch``     many uneven simulations advanced together, each read back
* ``serve``     requests through the continuous-batching server until all are done
* ``packed``    host-built packed tree uploaded, traversed, accelerations back
* ``probes``    FP64 direct sums at probe bodies (the stated force error)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from galaxy_b200 import presets, scenarios
from galaxy_b200.batch import Batch
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime, bodies_to_state
from galaxy_b200.serve import NativeServer


def listed() -> list[dict]:
    return [
        # the smallest simulation of the batched workload, alone: launch latency
        _evolve("evolve-disc-1k", "exponential_disc", 1024, 0.01, 0.5, 1, 1e-3, 50),
        # one galaxy of 16,384 bodies, 100 steps (the CPU-comparable workload)
        _evolve("evolve-disc-16k", "exponential_disc", 16384, 0.01, 0.5, 1, 1e-3, 100),
        # the headline: cold collapse of 2^20 bodies, a snapshot every 40 steps
        _evolve("evolve-cold-1m", "cold_disc", 1 << 20, 0.005, 0.5, 1, 5e-4, 40),
        # the same physics at the opening angle of 1e-3 force error, a ragged size
        _evolve("evolve-accurate-700k", "cold_disc", 700001, 0.005, 0.12, 1, 5e-4, 10),
        # precision form: binary encounter of 2^22 bodies, compensated sums
        _evolve("evolve-precise-4m", "binary_encounter", 1 << 22, 0.005, 0.5, 1, 5e-4, 20,
                compensated=True),
        # diagnostics of the precision form: forces with the potential, invariants
        {"name": "solve-precise-262k", "kind": "solve", "scenario": "binary_encounter",
         "n": 262147, "eps": 0.005, "theta": 0.7, "bucket": 4, "compensated": True,
         "potential": True},
        # the receipt tool's collision evolved by the reference's own call sequence
        {"name": "loop-collision-64k", "kind": "loop", "scenario": "collision", "n": 65536,
         "eps": 0.05, "theta": 0.5, "bucket": 4, "dt": 0.01, "steps": 8},
        # batched workload: 96 uneven simulations, 2^10 to 2^16 bodies each
        {"name": "batch-96", "kind": "batch", "count": 96, "lo": 10, "hi": 16, "eps": 0.01,
         "theta": 0.5, "bucket": 1, "dt": 1e-3, "steps": 20},
        # a burst of requests through the server
        {"name": "serve-12", "kind": "serve", "count": 12, "lo": 12, "hi": 18, "eps": 0.01,
         "theta": 0.5, "bucket": 1, "dt": 1e-3, "steps": 100},
        # host-tree path: packed records up, accelerations down
        {"name": "packed-131k", "kind": "packed", "scenario": "cold_disc", "n": 131071,
         "eps": 0.01, "theta": 0.5, "bucket": 1},
        # the force error of the headline workload at 4,096 probe bodies
        {"name": "probes-4096-of-1m", "kind": "probes", "scenario": "cold_disc", "n": 1 << 20,
         "eps": 0.005, "theta": 0.5, "bucket": 1, "probes": 4096},
    ]


def draw(rng) -> dict:
    """Another case of the same ranges: sizes over their logarithm, odd ones
    among them, the options in the shares a user meets them in."""
    kind = rng.choice(["evolve"] * 6 + ["solve"] * 3 + ["loop"] * 2 + ["batch"] * 2
                      + ["serve", "packed", "packed", "probes"])

    def size(lo, hi):
        return int(2.0 ** rng.uniform(lo, hi))

    scenario = rng.choice(["cold_disc", "exponential_disc", "binary_encounter"])
    case = {"kind": kind, "scenario": scenario, "eps": rng.choice([0.005, 0.01, 0.05]),
            "theta": round(rng.uniform(0.3, 0.8), 3), "bucket": rng.choice([1, 1, 1, 2, 4, 8, 16])}
    if kind == "evolve":
        n = size(10, 21)
        per_step = n * _terms(n, case["theta"])
        budget = (1 << 22) * 10 * _terms(1 << 22, 0.5)
        case.update(n=n, dt=rng.choice([5e-4, 1e-3]), compensated=rng.random() < 0.25,
                    steps=max(1, min(rng.randint(10, 60), int(budget / per_step))))
    elif kind == "solve":
        case.update(n=size(10, 20), compensated=rng.random() < 0.4,
                    potential=rng.random() < 0.4)
    elif kind == "loop":
        case.update(scenario=rng.choice(["disc", "collision"]), n=2 * size(11, 16), eps=0.05,
                    theta=0.5, bucket=rng.choice([1, 4]), dt=0.01, steps=rng.randint(2, 8))
    elif kind in ("batch", "serve"):
        del case["scenario"]
        case.update(count=rng.randint(8, 64) if kind == "batch" else rng.randint(4, 16),
                    lo=rng.randint(10, 12), hi=rng.randint(13, 16), dt=1e-3,
                    steps=rng.randint(5, 40))
    elif kind == "probes":
        case.update(n=size(12, 20), probes=int(2.0 ** rng.uniform(3.5, 12)))
    else:
        case.update(n=size(11, 18))
    return case


# ------------------------------------------------------------- preparation --


class _State:
    """What a program holds between calls: device, simulation, tree."""

    def __init__(self, case):
        self.case = case
        self.server = None

    def __del__(self):
        if self.server is not None:
            self.server.stop()


def prepare(case: dict, seed: int) -> _State:
    s = _State(case)
    kind = case["kind"]
    if kind == "serve":
        cfg = _config(case)
        s.server = NativeServer(budget_bytes=16 << 30, round_steps=16)
        s.requests = [(bodies_to_state(b), cfg, case["dt"], k)
                      for b, k in zip(_members(case, seed), _request_steps(case, seed))]
        return s
    s.gpu = NbodyGpu("0")
    if kind == "batch":
        s.states = [s.gpu.create_evolving_state(b)[0] for b in _members(case, seed)]
        s.batch = Batch(s.gpu, s.states, [_config(case)] * len(s.states))
        s.batch.solve()
        return s
    s.cfg = _config(case)
    s.rt = ParallelTreeRuntime(s.gpu)
    s.ev, _ = s.gpu.create_evolving_state(_bodies(case, seed))
    if kind == "probes":
        s.probes = _probe_indices(case, seed)
        return s
    s.tree = s.rt.create_tree(s.gpu, s.ev, s.cfg)
    s.rt.rebuild(s.gpu, s.ev, s.tree, s.cfg)
    if kind == "packed":
        s.packed = s.rt.read_evidence(s.gpu, s.tree).packed(s.cfg)
    elif kind in ("evolve", "loop"):
        s.rt.force(s.gpu, s.ev, s.tree, s.cfg)  # the boundary acceleration
    return s


def run(s: _State):
    case, kind = s.case, s.case["kind"]
    if kind == "serve":
        ids = [s.server.submit(*r) for r in s.requests]
        done = {}
        while len(done) < len(ids):
            got = s.server.poll(60.0)
            if got is None:
                raise RuntimeError("a request did not finish")
            done[got[0]["request_id"]] = got[1]
        return [_fields(done[i]) for i in ids]
    if kind == "batch":
        s.batch.step(case["dt"], case["steps"])
        got = [s.gpu.read_evolving_state_records(st)[0] for st in s.states]
        return _fields(np.concatenate(got))
    if kind == "probes":
        return s.gpu.direct_probes(s.ev, s.cfg, s.probes)
    if kind == "packed":
        return s.gpu.traverse(s.packed).accelerations
    if kind == "evolve":
        s.rt.step(s.gpu, s.ev, s.tree, s.cfg, case["dt"], case["steps"])
        return _fields(s.gpu.read_evolving_state_records(s.ev)[0])
    if kind == "loop":
        for _ in range(case["steps"]):
            s.gpu.kick_drift(s.ev, case["dt"])
            s.rt.rebuild(s.gpu, s.ev, s.tree, s.cfg)
            s.rt.force(s.gpu, s.ev, s.tree, s.cfg)
            s.gpu.final_kick(s.ev, case["dt"])
        return _fields(s.gpu.read_evolving_state_records(s.ev)[0])
    s.rt.rebuild(s.gpu, s.ev, s.tree, s.cfg)
    s.rt.force(s.gpu, s.ev, s.tree, s.cfg)
    accel = s.gpu.read_evolving_accelerations_f32(s.ev)[0]
    inv = s.gpu.conservation(s.ev)
    return {"accel": accel, "invariants": [inv[k] for k in _INVARIANTS]}


def work(case: dict) -> dict:
    """What a pass cannot do without.  Terms: about 10 / theta^1.5 per octave
    of the quadtree and body (2.8e2 at theta 0.5 and 2.4e3 at theta 0.12 for
    2^20 bodies), 20 operations each; records read and written once a step."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        sizes = _sizes(case, 1)
        steps = _request_steps(case, 1) if kind == "serve" else [case["steps"]] * len(sizes)
        return {"bytes": sum(96.0 * n * k + 32.0 * n for n, k in zip(sizes, steps)),
                "flops": sum(20.0 * n * k * _terms(n, case["theta"])
                             for n, k in zip(sizes, steps))}
    n = case["n"]
    if kind == "probes":
        return {"bytes": 32.0 * n + 16.0 * case["probes"], "flops": 20.0 * n * case["probes"]}
    force = 20.0 * n * _terms(n, case["theta"])
    if kind == "packed":  # 32 + 16 bytes a body and 64 a cell in, 16 a body out
        return {"bytes": n * (64.0 + 64.0 * 1.75 / case["bucket"] ** 0.5), "flops": force}
    if kind == "solve":
        return {"bytes": 48.0 * n, "flops": force}
    return {"bytes": 96.0 * n * case["steps"] + 32.0 * n, "flops": force * case["steps"]}


def exact(case: dict, seed: int):
    """The same results in 64 bits by plain torch: state held in the f32
    records between kicks and drifts, as the format demands, everything else
    in f64.  None where the steps would take too long."""
    kind = case["kind"]
    if kind == "serve":
        return None
    if kind == "batch":
        sizes = _sizes(case, seed)
        if case["steps"] * sum(_cost(n, case["theta"]) for n in sizes) > 10.0:
            return None
        got = [_evolved(b, case, case["steps"]) for b in _members(case, seed)]
        return {k: np.concatenate([g[k] for g in got]) for k in got[0]}
    bodies = _bodies(case, seed)
    state = _records(bodies)
    if kind == "probes":
        return _direct(state, case, _probe_indices(case, seed))
    if kind in ("evolve", "loop"):
        if case["steps"] * _cost(case["n"], case["theta"]) > 10.0:
            return None
        return _evolved(bodies, case, case["steps"])
    if _cost(case["n"], case["theta"]) > 10.0:
        return None
    acc, phi = _tree_force(state, case)
    if kind == "packed":
        return acc.cpu().numpy()
    x, y, m, vx, vy = state
    accel = torch.zeros(len(x), 4, dtype=torch.float64, device=x.device)
    accel[:, :2] = acc
    mass = m.sum()
    kinetic = (0.5 * m * (vx * vx + vy * vy)).sum()
    potential = (0.5 * m * phi).sum() if case["potential"] else torch.zeros_like(mass)
    inv = {"mass": mass, "com_x": (m * x).sum() / mass, "com_y": (m * y).sum() / mass,
           "kinetic": kinetic, "potential": potential, "energy": kinetic + potential}
    return {"accel": accel.cpu().numpy(), "invariants": [float(inv[k]) for k in _INVARIANTS]}


# ------------------------------------------------------------------ inputs --

_INVARIANTS = ("mass", "com_x", "com_y", "kinetic", "potential", "energy")


def _evolve(name, scenario, n, eps, theta, bucket, dt, steps, compensated=False) -> dict:
    return {"name": name, "kind": "evolve", "scenario": scenario, "n": n, "eps": eps,
            "theta": theta, "bucket": bucket, "dt": dt, "steps": steps,
            "compensated": compensated}


def _config(case) -> Config:
    return Config(theta=case["theta"], softening_kpc=case["eps"], g=_g(case),
                  bucket=case["bucket"], compensated=bool(case.get("compensated")),
                  potential=bool(case.get("potential")))


def _g(case) -> float:
    return Config().g if case.get("scenario") in ("disc", "collision") else 1.0


def _bodies(case, seed) -> np.ndarray:
    if case["scenario"] == "disc":
        return presets.make_disc(case["n"], seed)
    if case["scenario"] == "collision":
        return presets.make_collision(case["n"], seed)
    return scenarios.make(case["scenario"], case["n"], seed, case["eps"])


def _sizes(case, seed) -> list[int]:
    """Members log-uniform in [2^lo, 2^hi], one at each end.  The sizes are the
    case's own, the same for every seed."""
    rng = np.random.default_rng(case["count"] * 1000 + case["lo"] * 50 + case["hi"])
    n = 2.0 ** rng.uniform(case["lo"], case["hi"], case["count"])
    n[0], n[-1] = 2 ** case["lo"], 2 ** case["hi"]
    return [int(v) for v in n]


def _members(case, seed) -> list[np.ndarray]:
    names = list(scenarios.SCENARIOS)
    return [scenarios.make(names[i % 3], n, seed * 1000 + i, case["eps"])
            for i, n in enumerate(_sizes(case, seed))]


def _request_steps(case, seed) -> list[int]:
    """Steps log-uniform in [10, steps], fixed by the case."""
    rng = np.random.default_rng(case["count"] * 77 + case["steps"])
    lo, hi = math.log(min(10, case["steps"])), math.log(case["steps"])
    return [int(round(math.exp(v))) for v in rng.uniform(lo, hi, case["count"])]


def _probe_indices(case, seed) -> np.ndarray:
    k = min(case["probes"], case["n"])
    return np.random.default_rng(seed).choice(case["n"], k, replace=False).astype(np.uint32)


def _fields(records: np.ndarray) -> dict:
    return {"position_mass": records["position_mass"], "velocity": records["velocity"]}


def _terms(n, theta) -> float:
    """Interactions per body, about."""
    return min(float(n), 10.0 / theta ** 1.5 * max(1.0, math.log(n, 4)))


def _cost(n, theta) -> float:
    """Seconds of one f64 force below, about."""
    return 0.02 + 6e-9 * n * _terms(n, theta)


# --------------------------------------------------------- 64-bit reference --


def _records(bodies):
    """x, y, mass, vx, vy of the f32 records, in f64 on the GPU."""
    t = torch.from_numpy(np.ascontiguousarray(bodies[:, [0, 1, 4, 2, 3]])).to("cuda")
    return [c.contiguous() for c in t.to(torch.float32).to(torch.float64).T]


def _f32(v):
    return v.to(torch.float32).to(torch.float64)


def _evolved(bodies, case, steps) -> dict:
    x, y, m, vx, vy = _records(bodies)
    dt = float(np.float32(case["dt"]))
    acc, _ = _tree_force([x, y, m], case)
    for _ in range(steps):
        vx, vy = _f32(vx + 0.5 * dt * acc[:, 0]), _f32(vy + 0.5 * dt * acc[:, 1])
        x, y = _f32(x + dt * vx), _f32(y + dt * vy)
        acc, _ = _tree_force([x, y, m], case)
        vx, vy = _f32(vx + 0.5 * dt * acc[:, 0]), _f32(vy + 0.5 * dt * acc[:, 1])
    zero = torch.zeros_like(x)
    return {"position_mass": torch.stack([x, y, m, zero], 1).cpu().numpy(),
            "velocity": torch.stack([vx, vy, zero, zero], 1).cpu().numpy()}


def _spread(v):
    for s, k in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << s)) & k
    return v


def _morton(v, center, half):
    q = torch.floor((v - (center - half)) / (half * 2.0) * 65536.0)
    return _spread(q.clamp(0.0, 65535.0).to(torch.int64))


def _tree_force(state, case):
    """Barnes-Hut accelerations and potential in f64: quadtree of 32-bit Morton
    codes, a cell is a point mass when it does not hold the body and
    width / distance < theta, leaves are summed body by body."""
    x, y, m = state[:3]
    n, dev = len(x), x.device
    lo_x, hi_x, lo_y, hi_y = (float(v) for v in (x.min(), x.max(), y.min(), y.max()))
    span = max(hi_x - lo_x, hi_y - lo_y, 1e-12)
    half = span * 0.500000000001 + 1e-12
    code = _morton(x, (lo_x + hi_x) * 0.5, half) | (_morton(y, (lo_y + hi_y) * 0.5, half) << 1)
    code, order = torch.sort(code, stable=True)
    sx, sy, sm = x[order], y[order], m[order]
    cells, first = [], 0
    live = torch.ones(n, dtype=torch.bool, device=dev)  # positions whose cell was split
    for depth in range(17):
        at = torch.nonzero(live).squeeze(1)
        if not len(at):
            break
        key, inverse, count = torch.unique_consecutive(
            code[at] >> (32 - 2 * depth), return_inverse=True, return_counts=True)
        start = at[torch.cumsum(count, 0) - count]
        mass, wx, wy = (torch.zeros(len(count), dtype=torch.float64, device=dev).index_add_(
            0, inverse, v[at]) for v in (sm, sm * sx, sm * sy))
        leaf = (count <= case["bucket"]) | (depth == 16)
        cells.append([start, count, wx / mass, wy / mass, mass, leaf,
                      torch.full_like(mass, half * 0.5 ** depth * 2.0), key])
        live = torch.zeros(n, dtype=torch.bool, device=dev)
        live[at] = ~leaf[inverse]
    # children of the split cells of one depth are the cells of the next, in order
    for d, c in enumerate(cells):
        first += len(c[0])
        nch = torch.zeros_like(c[0])
        if d + 1 < len(cells):
            split = torch.nonzero(~c[5]).squeeze(1)
            nch[split] = torch.unique_consecutive(cells[d + 1][7] >> 2, return_counts=True)[1]
        c += [nch, first + torch.cumsum(nch, 0) - nch]
    start, count, cx, cy, cm, leaf, width, _, nch, child = (torch.cat(v) for v in zip(*cells))
    eps2, g = float(np.float32(case["eps"])) ** 2, _g(case)
    g = float(np.float32(g))
    out = torch.zeros(n, 3, dtype=torch.float64, device=dev)

    def add(i, dx, dy, mass):
        inv = 1.0 / torch.sqrt(dx * dx + dy * dy + eps2)
        s = g * mass * inv * inv * inv
        out.index_add_(0, i, torch.stack([dx * s, dy * s, -g * mass * inv], 1))

    def spread(i, k, begin):
        """Each i repeated k times, beside begin, begin + 1, ..."""
        r = torch.repeat_interleave(i, k)
        base = torch.repeat_interleave(begin - (torch.cumsum(k, 0) - k), k)
        return r, base + torch.arange(len(r), device=dev)

    for p0 in range(0, n, 1 << 16):
        i = torch.arange(p0, min(n, p0 + (1 << 16)), device=dev)
        c = torch.zeros_like(i)
        while len(i):
            isleaf = leaf[c]
            li, lb = spread(i[isleaf], count[c[isleaf]], start[c[isleaf]])
            other = li != lb
            li, lb = li[other], lb[other]
            add(li, sx[lb] - sx[li], sy[lb] - sy[li], sm[lb])
            i, c = i[~isleaf], c[~isleaf]
            dx, dy = cx[c] - sx[i], cy[c] - sy[i]
            dist = torch.sqrt(dx * dx + dy * dy)
            holds = (i >= start[c]) & (i < start[c] + count[c])
            point = ~holds & (dist > 0) & (width[c] / dist < case["theta"])
            add(i[point], dx[point], dy[point], cm[c[point]])
            i, c = i[~point], c[~point]
            i, c = spread(i, nch[c], child[c])
    back = torch.empty_like(out)
    back[order] = out
    return back[:, :2], back[:, 2]


def _direct(state, case, probes):
    """FP64 direct sums at the probe bodies."""
    x, y, m = state[:3]
    p = torch.from_numpy(probes.astype(np.int64)).to(x.device)
    out = []
    for k in range(0, len(p), 64):
        q = p[k:k + 64]
        dx, dy = x[None] - x[q, None], y[None] - y[q, None]
        inv = 1.0 / torch.sqrt(dx * dx + dy * dy + case["eps"] ** 2)
        s = _g(case) * m[None] * inv * inv * inv
        s[torch.arange(len(q)), q] = 0.0
        out.append(torch.stack([(dx * s).sum(1), (dy * s).sum(1)], 1))
    return torch.cat(out).cpu().numpy()
