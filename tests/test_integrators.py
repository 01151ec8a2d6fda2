"""The kernels that sum partials, at the edges of their splits: batches just below
and above the size up to which four threads share a body (32768), where a
batch's steps and gradients must be those of its systems stepped by themselves
or in a small batch within the FP32 bounds of the pair terms (each side 2e-5
(|a| + mean|a|) off the oracle, gradients 1e-4 in norm), FP64 batches within
1e-13; the compensated integrator around rows of 384 bodies and more than eight
of them within 2e-5 of the oracle."""
import numpy as np
import pytest

import oracle
from utc_gb300 import ics
from utc_gb300.nbody import NBodyBatch, NBodySystem

pytestmark = pytest.mark.gpu

EPS2, DT = float(np.float32(1e-3)), float(np.float32(2 ** -10))
HEAD = [1, 2, 31, 33, 383, 384, 385, 3000]


def _sizes(total):
    left = total - sum(HEAD)
    return HEAD + [4096] * (left // 4096) + ([left % 4096] if left % 4096 else [])


def _states(sizes):
    states = [ics.uniform_cube(n, seed=n) for n in sizes]
    return np.concatenate([p for p, _ in states]), np.concatenate([v * 0 for _, v in states])


@pytest.mark.parametrize("precision,bound", [("f32", 4e-5), ("f64", 2e-13)])
@pytest.mark.parametrize("total", [32767, 32768, 32769, 65537])
def test_batch_against_its_systems(cuda, precision, bound, total):
    sizes = _sizes(total)
    pos, vel = _states(sizes)
    if precision == "f32":
        pos, vel = ics.f32(pos), ics.f32(vel)
    got = []
    for alone in (False, True):
        with NBodyBatch(sizes, precision=precision, kick="physical", eps2=EPS2, damping=1.0, dt=DT) as b:
            b.set_state(pos, vel)
            b.step_per_system(1) if alone else b.step(1)
            got.append(b.get_state())
    o = 0
    for n in sizes:  # from rest, so the velocities are the accelerations times dt
        a, b = (g[1][o:o + n, :3].astype(np.float64) for g in got)
        w = np.linalg.norm(b, axis=1)
        assert (np.linalg.norm(a - b, axis=1) <= bound * (w + w.mean())).all(), n
        o += n
    assert got[0][0][:, 3].tobytes() == pos[:, 3].tobytes()


def test_batch_gradients_do_not_depend_on_its_size(cuda):
    import torch

    got = []
    for total in (32768, 36865):  # the larger one holds the same systems and one more
        sizes = _sizes(32768) + ([total - 32768] if total > 32768 else [])
        pos, vel = _states(sizes)
        with NBodyBatch(sizes, kick="physical", eps2=EPS2, damping=1.0, dt=DT) as b:
            b.set_state(ics.f32(pos), ics.f32(vel))
            b.adj_forward(3, 2)
            gx = torch.zeros((b.nbody, 4), device="cuda")
            gx[:, :3] = torch.from_numpy(np.random.default_rng(1).normal(size=(36865, 3))[:b.nbody].astype(np.float32))
            got.append([t.cpu().numpy()[:32768] for t in b.adj_backward(gx)])
    o = 0
    for n in _sizes(32768):
        for x, y in zip(*got):
            d = np.linalg.norm((x[o:o + n] - y[o:o + n]).astype(np.float64))
            assert d <= 2e-4 * np.linalg.norm(y[o:o + n].astype(np.float64)) + 1e-12
        o += n


@pytest.mark.parametrize("n", [1, 31, 33, 383, 384, 385, 3071, 3073, 3457, 7000])
def test_compensated_integrator(cuda, n):
    pos, vel = _states([n])
    pos, vel = ics.f32(pos).astype(np.float64), vel.astype(np.float64)
    with NBodySystem(n, "f32comp", "sym", kick="physical", eps2=EPS2, damping=1.0, dt=DT) as s:
        s.set_state(pos, vel)
        a = s.accel()[:, :3]
        s.step(1)
        p, v = s.get_state()
    ref = oracle.accel(pos, EPS2)[:, :3]
    w = np.linalg.norm(ref, axis=1)
    bound = 2e-5 * (w + w.mean())
    assert (np.linalg.norm(a - ref, axis=1) <= bound).all()
    assert (np.linalg.norm(v[:, :3] - ref * DT, axis=1) <= bound * DT).all()
    assert np.abs(p[:, :3] - pos[:, :3] - v[:, :3] * DT).max() <= 2.0 ** -51
