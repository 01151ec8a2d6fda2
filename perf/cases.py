"""The work that is timed when this library is made faster: one case per way in which a program uses it.

A case is a dict of plain values; `prepare` makes what a program has in hand before the call (device or host arrays
and the context that it keeps), `run` is one pass through the public entry points, `exact` is the same pass in
64-bit torch, and `work` what the pass cannot do without.  Sizes are those of the configurations in bench.py and
the tests (N = 1024 of the reference app, 4096 of its multi-task app, 16384, 65536, 131072, 1048576, the batch of
512 systems of 128 to 16384 bodies), with ragged ones among them.
"""
import math

import numpy as np
import torch

from utc_gb300 import _native
from utc_gb300.nbody import NBodyBatch, NBodySystem, gpu_initial_conditions

#: 64-bit pair evaluations that exact() takes on; a larger case has no exact values.
EXACT_PAIRS = 1.3e11


def listed():
    return [
        # a program that looks at the state after every step (a viewer, an outer integrator): one launch pair
        {"name": "step1-n1024", "kind": "step", "n": 1024, "precision": "f32", "algo": "sym", "kick": "physical", "steps": 1, "start": "plummer"},
        # the reference app's own run (-n 1024 -l 100 -o 10) from host buffers, ten frames out
        {"name": "host100-n1024", "kind": "host", "n": 1024, "precision": "f32", "steps": 100, "every": 10},
        # a run of a small ragged system with the reference's kick
        {"name": "run50-n4099", "kind": "step", "n": 4099, "precision": "f32", "algo": "sym", "kick": "reference", "steps": 50, "start": "cube"},
        # the directed kernel: what NBodySystem and nb_params_default choose, and what a target shard steps with
        {"name": "fast20-n12345", "kind": "step", "n": 12345, "precision": "f32", "algo": "fast", "kick": "physical", "steps": 20, "start": "plummer"},
        # the GPU-scale forward run of the default bench line
        {"name": "run10-n65536", "kind": "step", "n": 65536, "precision": "f32", "algo": "sym", "kick": "physical", "steps": 10, "start": "plummer"},
        # the largest forward configuration
        {"name": "run1-n1048576", "kind": "step", "n": 1048576, "precision": "f32", "algo": "sym", "kick": "physical", "steps": 1, "start": "plummer"},
        # double state, the app's default type
        {"name": "f64-2-n16384", "kind": "step", "n": 16384, "precision": "f64", "algo": "sym", "kick": "reference", "steps": 2, "start": "plummer"},
        # the precision study: compensated forces, FP64 positions
        {"name": "comp2-n131071", "kind": "step", "n": 131071, "precision": "f32comp", "algo": "sym", "kick": "physical", "steps": 2, "start": "plummer"},
        # forward with checkpoints and the reverse pass
        {"name": "grad20-n16384", "kind": "grad", "n": 16384, "kick": "physical", "steps": 20, "every": 5},
        # the batch of 512 uneven systems
        {"name": "batch512-f32", "kind": "batch", "precision": "f32", "nsys": 512, "lo": 128, "hi": 16384, "steps": 4},
        # energy, momentum and per-body potentials of a state (a run's diagnostics)
        {"name": "energy-n65536", "kind": "energy", "n": 65536, "precision": "f32", "algo": "sym"},
        # bodies drawn on the GPU
        {"name": "ics-plummer-1m", "kind": "ics", "n": 1048576, "start": "plummer", "precision": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "host", "grad", "batch", "energy", "ics"])
    if kind == "step":
        precision, algo, hi = rng.choice([("f32", "sym", 1000000), ("f32", "sym", 100000), ("f32", "fast", 130000),
                                          ("f64", "sym", 65000), ("f32comp", "sym", 260000)])
        n = _log_int(rng, 500, hi)
        most = {"f32": 5e10, "f64": 2.5e9, "f32comp": 4e10}[precision]
        steps = max(1, min(_log_int(rng, 1, 100), int(most / (float(n) * n))))
        return {"kind": kind, "n": n, "precision": precision, "algo": algo, "kick": rng.choice(["physical", "reference"]),
                "steps": steps, "start": rng.choice(["plummer", "cube"])}
    if kind == "host":
        every = rng.randint(1, 20)
        return {"kind": kind, "n": _log_int(rng, 500, 20000), "precision": rng.choice(["f32", "f64"]),
                "steps": every * rng.randint(2, 6) + rng.randint(0, 3), "every": every}
    if kind == "grad":
        n = _log_int(rng, 700, 40000)
        return {"kind": kind, "n": n, "kick": rng.choice(["physical", "reference"]), "steps": rng.randint(3, 20), "every": rng.randint(1, 7)}
    if kind == "batch":
        precision = rng.choice(["f32", "f32", "f64"])
        lo = _log_int(rng, 64, 1000)
        hi = _log_int(rng, 2 * lo, 16384 if precision == "f32" else 4096)
        return {"kind": kind, "precision": precision, "nsys": _log_int(rng, 8, 400), "lo": lo, "hi": hi, "steps": rng.randint(1, 5)}
    if kind == "energy":
        precision, hi = rng.choice([("f32", 150000), ("f64", 32000), ("f32comp", 100000)])
        return {"kind": kind, "n": _log_int(rng, 1000, hi), "precision": precision, "algo": "sym"}
    return {"kind": kind, "n": _log_int(rng, 5000, 8000000), "start": rng.choice(["plummer", "plummer", "cube", "shell"]),
            "precision": rng.choice(["f32", "f64"])}


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _f32(x):
    return float(np.float32(x))


def _params(case):
    """eps2, damping, dt, G and the masses' scale; floats, so that every precision takes the same values."""
    if case.get("kick") == "reference":  # the app's: unit masses, its softening and damping
        return {"eps2": _f32(0.00125), "damping": _f32(0.995), "dt": 2.0 ** -16, "G": 1.0}
    return {"eps2": 2.0 ** -13, "damping": 1.0, "dt": 2.0 ** -13, "G": 1.0}


def _directions(rng, r):
    c = rng.uniform(-1.0, 1.0, r.size)
    f = rng.uniform(0.0, 2.0 * math.pi, r.size)
    s = np.sqrt(1.0 - c * c)
    return np.stack([r * s * np.cos(f), r * s * np.sin(f), r * c], axis=1)


def _bodies(n, start, rng, unit_masses):
    """(n, 4) positions and velocities in float64: a Plummer sphere (virial units) or a uniform cube."""
    pos, vel = np.empty((n, 4)), np.empty((n, 4))
    if start == "plummer":
        r = 1.0 / np.sqrt(np.maximum(rng.uniform(0.0, 0.999, n), 1e-9) ** (-2.0 / 3.0) - 1.0)
        q = np.sqrt(rng.beta(1.5, 4.5, n))  # q^2 (1 - q^2)^(7/2), the isotropic speeds
        pos[:, :3] = _directions(rng, r)
        vel[:, :3] = _directions(rng, q * math.sqrt(2.0) * (1.0 + r * r) ** -0.25)
        pos[:, 3] = 1.0 / n
    else:
        pos[:, :3] = rng.uniform(-1.0, 1.0, (n, 3))
        vel[:, :3] = rng.uniform(-0.01, 0.01, (n, 3))
        pos[:, 3] = rng.uniform(0.5, 1.5, n) / n
    if unit_masses:
        pos[:, 3] *= n
    vel[:, 3] = 1.0
    return pos, vel


def _sizes(case):
    """Log-uniform system sizes in [lo, hi], spread by the golden ratio: the case alone gives them."""
    u = np.modf((np.arange(case["nsys"]) + 1) * 0.6180339887498949)[0]
    return np.clip(np.floor(case["lo"] * (case["hi"] / case["lo"]) ** u), case["lo"], case["hi"]).astype(np.int64)


def _host_inputs(case, seed):
    """The pass's inputs as float64 (n, 4) arrays that the case's own type holds exactly."""
    rng = np.random.default_rng(seed)
    unit = case.get("kick") == "reference" or case["kind"] == "host"
    if case["kind"] == "batch":
        parts = [_bodies(int(n), "plummer", rng, False) for n in _sizes(case)]
        pos, vel = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    else:
        pos, vel = _bodies(case["n"], case.get("start", "cube" if case["kind"] == "grad" else "plummer"), rng, unit)
    if case.get("precision", "f32") == "f32":
        pos, vel = pos.astype(np.float32).astype(np.float64), vel.astype(np.float32).astype(np.float64)
    more = ()
    if case["kind"] == "grad":  # cotangents of the final positions and velocities
        g = np.zeros((2, case["n"], 4))
        g[:, :, :3] = rng.normal(0.0, 1.0, (2, case["n"], 3))
        more = (g[0].astype(np.float32).astype(np.float64), g[1].astype(np.float32).astype(np.float64))
    return (pos, vel) + more


def _case_params(case):
    return _params({"kick": "reference"} if case["kind"] == "host" else case)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ics":
        return {"case": case, "seed": int(seed) + 1}
    q = _case_params(case)
    wide = case.get("precision", "f32") != "f32"
    dt = torch.float64 if wide else torch.float32
    arrays = _host_inputs(case, seed)
    st = {"case": case}
    if kind == "host":
        nt = np.float64 if wide else np.float32
        st["in"] = tuple(a.astype(nt) for a in arrays)
        st["sys"] = NBodySystem(case["n"], case["precision"], "sym", kick="reference", **q)
        return st
    st["in"] = tuple(torch.from_numpy(a).to(device="cuda", dtype=dt) for a in arrays)
    st["out"] = (torch.empty_like(st["in"][0]), torch.empty_like(st["in"][1]))
    if kind == "batch":
        st["sys"] = NBodyBatch(_sizes(case), precision=case["precision"], algo="sym", kick="physical", **q)
        st["stream"] = torch.cuda.Stream()
    else:
        st["sys"] = NBodySystem(case["n"], case.get("precision", "f32"), case.get("algo", "sym"), kick=case.get("kick", "physical"), **q)
    if kind == "energy":
        st["sys"].set_state(*st["in"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ics":
        return gpu_initial_conditions(case["start"], case["n"], seed=st["seed"], precision=case["precision"])
    s = st["sys"]
    if kind == "host":
        frames, _ = s.run_host(*st["in"], case["steps"], case["every"])
        return frames
    if kind == "energy":
        e, bodies = s.energy(with_bodies=True)
        return [e, bodies]
    if kind == "batch":
        stream, now = st["stream"], torch.cuda.current_stream()
        stream.wait_stream(now)
        with torch.cuda.stream(stream):
            s.set_state(*st["in"])
            s.run(case["steps"], stream.cuda_stream)
            p, v = st["out"]
            _native.check(s.lib.nb_batch_get_state(s.handle, p.data_ptr(), v.data_ptr(), _native.NB_DEVICE, stream.cuda_stream))
        now.wait_stream(stream)
        return list(st["out"])
    s.set_state(st["in"][0], st["in"][1])
    if kind == "step":
        s.step(case["steps"])
        s.get_state_device(*st["out"])
        return list(st["out"])
    s.adj_forward(case["steps"], case["every"])
    s.get_state_device(*st["out"])
    return list(st["out"]) + list(s.adj_backward(st["in"][2], st["in"][3]))


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def work(case):
    """Flops: each unordered pair once, 26 (three differences, the squared distance, one reciprocal square root, its
    cube, two weights, six multiply-adds); 30 with the potential of both bodies; the adjoint's pair term 60 on top."""
    wide = 2 if case.get("precision", "f32") != "f32" else 1
    kind = case["kind"]
    if kind == "ics":
        return {"bytes": 32.0 * wide * case["n"], "flops": 40.0 * case["n"]}
    n2 = float((_sizes(case).astype(float) ** 2).sum()) if kind == "batch" else float(case["n"]) ** 2
    n = float(_sizes(case).sum()) if kind == "batch" else float(case["n"])
    if kind == "energy":
        return {"bytes": 48.0 * wide * n, "flops": 15.0 * n2}
    if kind == "host":
        return {"bytes": 16.0 * wide * n * (2 + case["steps"] // case["every"]), "flops": 13.0 * n2 * case["steps"]}
    if kind == "grad":
        return {"bytes": 132.0 * n, "flops": (13.0 + 30.0) * n2 * case["steps"]}
    return {"bytes": 64.0 * wide * n, "flops": 13.0 * n2 * case["steps"]}


# ---------------------------------------------------------------------------------------------------------------
# the same passes in 64-bit torch
# ---------------------------------------------------------------------------------------------------------------
def _accel(x, m, eps2, potential=False):
    """Accelerations (n, 3) of bodies at x (n, 3), and the potentials over j != i, in row chunks."""
    n = x.shape[0]
    acc, phi = torch.empty_like(x), torch.empty_like(m)
    rows = max(1, min(n, 30_000_000 // n))
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [x[None, :, k] - x[a:b, None, k] for k in range(3)]
        inv = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2).rsqrt_()
        if potential:
            phi[a:b] = inv @ m - m[a:b] / math.sqrt(eps2)
        w = inv * inv * inv * m
        for k in range(3):
            acc[a:b, k] = (w * d[k]).sum(1)
    return (acc, phi) if potential else acc


def _step(x, v, m, q, kick):
    k = m[:, None] if kick == "reference" else q["G"]
    v = (v + _accel(x, m, q["eps2"]) * k * q["dt"]) * q["damping"]
    return x + v * q["dt"], v


def _state(x, v, m):
    return [torch.cat([x, m[:, None]], 1), torch.cat([v, torch.ones_like(m)[:, None]], 1)]


def _grad_exact(x, v, m, gx, gv, case, q):
    xs, steps, kick = [x], case["steps"], case["kick"]
    for _ in range(steps):
        x, v = _step(x, v, m, q, kick)
        xs.append(x)
    final = _state(x, v, m)
    gm = torch.zeros_like(m)
    n, rows = m.numel(), max(1, min(m.numel(), 8_000_000 // m.numel()))
    for t in range(steps - 1, -1, -1):
        mu = (gv + q["dt"] * gx) * q["damping"]  # the cotangent of the kicked velocity
        gv = mu
        xt = xs[t].clone().requires_grad_(True)
        mt = m.clone().requires_grad_(True)
        for a in range(0, n, rows):
            b = min(n, a + rows)
            r = xt[None, :, :] - xt[a:b, None, :]
            w = mt * (r.square().sum(2) + q["eps2"]).pow(-1.5)
            acc = (w[:, :, None] * r).sum(1)
            k = mt[a:b, None] if kick == "reference" else q["G"]
            dx, dm = torch.autograd.grad((acc * k * q["dt"] * mu[a:b]).sum(), (xt, mt))
            gx = gx + dx
            gm = gm + dm
    zero = torch.zeros_like(m)[:, None]
    return final + [torch.cat([gx, zero], 1), torch.cat([gv, zero], 1), gm]


def _u64(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _splitmix(z):
    """The SplitMix64 finaliser on int64 tensors (two's complement stands for unsigned)."""
    z = z + _u64(0x9E3779B97F4A7C15)
    for shift, mult in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB)):
        z = (z ^ ((z >> shift) & ((1 << (64 - shift)) - 1))) * _u64(mult)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _ics_exact(case, seed):
    n, start = case["n"], case["start"]
    ids = torch.arange(n, dtype=torch.int64, device="cuda")

    def u(k):  # stream k of every body: 53 random bits
        h = _splitmix(_splitmix(ids * 256 + k) ^ seed)
        return ((h >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53

    one = torch.ones(n, dtype=torch.float64, device="cuda")
    if start == "cube":
        p = [2 * u(0) - 1, 2 * u(1) - 1, 2 * u(2) - 1, (0.5 + u(3)) / n]
        v = [0.01 * (2 * u(k) - 1) for k in (4, 5, 6)] + [one]
        return [torch.stack(p, 1), torch.stack(v, 1)]
    if start == "shell":
        x, todo = [one.clone() for _ in range(3)], torch.ones(n, dtype=torch.bool, device="cuda")
        for t in range(40):
            c = [2 * u(8 + 3 * t + k) - 1 for k in range(3)]
            for k in range(3):
                x[k] = torch.where(todo, c[k], x[k])
            todo = todo & (c[0] * c[0] + c[1] * c[1] + c[2] * c[2] > 1)
            if not bool(todo.any()):
                break
        length = torch.sqrt(x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
        x = [c / length for c in x]
        p = [x[k] * (2.5 + 1.5 * u(128 + k)) for k in range(3)]
        il = 1.0 / torch.sqrt(x[0] ** 2 + x[1] ** 2 + 1)
        near = 1 - x[2] < 1e-6
        ax = [torch.where(near, x[1] * il, 0 * one), torch.where(near, x[0] * il, 0 * one), torch.where(near, il, one)]
        v = [(p[1] * ax[2] - p[2] * ax[1]) * 0.01, (p[2] * ax[0] - p[0] * ax[2]) * 0.01, (p[0] * ax[1] - p[1] * ax[0]) * 0.01, one]
        return [torch.stack(p + [one], 1), torch.stack(v, 1)]
    r = 1.0 / torch.sqrt((0.999 * u(0)).clamp(min=1e-300).pow(-2.0 / 3.0) - 1)

    def sphere(length, kc, kf):
        c = 2 * u(kc) - 1
        s = torch.sqrt((1 - c * c).clamp(min=0))
        f = 2 * math.pi * u(kf)
        return torch.stack([length * s * f.cos(), length * s * f.sin(), length * c], 1)

    q, todo = 0 * one + math.sqrt(2.0 / 9.0), torch.ones(n, dtype=torch.bool, device="cuda")
    for t in range(64):
        a, b = u(8 + 2 * t), 0.1 * u(9 + 2 * t)
        ok = todo & (b < a * a * (1 - a * a).pow(3.5))
        q = torch.where(ok, a, q)
        todo = todo & ~ok
        if not bool(todo.any()):
            break
    p, v = sphere(r, 1, 2), sphere(q * math.sqrt(2.0) * (r * r + 1).pow(-0.25), 3, 4)
    p, v = p - p.mean(0), v - v.mean(0)
    return [torch.cat([p, one[:, None] / n], 1), torch.cat([v, one[:, None]], 1)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ics":
        return _ics_exact(case, int(seed) + 1)
    n2 = float((_sizes(case).astype(float) ** 2).sum()) if kind == "batch" else float(case["n"]) ** 2
    if n2 * case.get("steps", 1) * (4 if kind == "grad" else 1) > EXACT_PAIRS:
        return None
    q = _case_params(case)
    ins = [torch.from_numpy(a).cuda() for a in _host_inputs(case, seed)]
    x, m, v = ins[0][:, :3].contiguous(), ins[0][:, 3].contiguous(), ins[1][:, :3].contiguous()
    if kind == "grad":
        return _grad_exact(x, v, m, ins[2][:, :3], ins[3][:, :3], case, q)
    if kind == "energy":
        acc, phi = _accel(x, m, q["eps2"], True)
        p = (m[:, None] * v).sum(0)
        e = torch.stack([0.5 * (m * v.square().sum(1)).sum(), -0.5 * q["G"] * (m * phi).sum(), p[0], p[1], p[2]])
        return [e, torch.cat([acc, phi[:, None]], 1)]
    if kind == "host":
        frames = []
        for t in range(case["steps"]):
            x, v = _step(x, v, m, q, "reference")
            if (t + 1) % case["every"] == 0:
                frames.append(_state(x, v, m)[0])
        return torch.stack(frames)
    offs = np.concatenate([[0], np.cumsum(_sizes(case))]) if kind == "batch" else [0, case["n"]]
    for a, b in zip(offs[:-1], offs[1:]):
        for _ in range(case["steps"]):
            x[a:b], v[a:b] = _step(x[a:b].clone(), v[a:b].clone(), m[a:b], q, case.get("kick", "physical"))
    return _state(x, v, m)
