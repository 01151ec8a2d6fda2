"""Directed plans of the automatic shape up to 24576 bodies sum every target in one
CTA (utc_gb300/csrc/nb_small.cu) and integrate in a second launch: at the edges
of its tiles and of the rule accelerations within 2e-5 (|a| + mean|a|) of the
FP64 oracle, as of the stream-K kernel that other shapes run; the plan given
explicitly, graph replay and shards of the targets give the same bits."""
import numpy as np
import pytest

import oracle
from test_shard_gpu import run_shards
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

pytestmark = pytest.mark.gpu

EPS2, DT = float(np.float32(1e-3)), float(np.float32(1e-3))


def _states(n, pos, vel, **kw):
    with NBodySystem(n, "f32", "fast", kick="reference", eps2=EPS2, damping=1.0, dt=DT, **kw) as s:
        assert s.launches_per_step() == 2
        info = s.plan_info()
        s.set_state(pos, vel)
        a = s.accel()
        s.step(1)
        one = s.get_state()
        s.step(33)
        return info, a, one, s.get_state()


@pytest.mark.parametrize("n", [1, 2, 3, 7, 127, 129, 1999, 2000, 2049, 8191, 8192, 8999, 9000, 9001, 24575, 24576, 24577])
def test_direct_vs_oracle_and_other_shapes(cuda, n):
    p, v = ics.uniform_cube(n, seed=n)
    pos, vel = ics.f32(p), ics.f32(v)
    info, a, one, many = _states(n, pos, vel)
    _, a2, one2, many2 = _states(n, pos, vel, block=info["block"], bpt=info["bpt"])  # the same plan
    other = _states(n, pos, vel, block=256, bpt=4)  # never the automatic shape
    assert a.tobytes() == a2.tobytes()
    for k in range(2):
        assert one[k].tobytes() == one2[k].tobytes() and many[k].tobytes() == many2[k].tobytes()
    with NBodySystem(n, "f32", "fast", kick="reference", eps2=EPS2, damping=1.0, dt=DT) as s:
        s.set_state(pos, vel)
        for _ in range(34):
            s.step(1)
        single = s.get_state()
    assert single[0].tobytes() == many[0].tobytes() and single[1].tobytes() == many[1].tobytes()
    ref = oracle.accel(pos.astype(np.float64), EPS2)[:, :3]
    w = np.linalg.norm(ref, axis=1)
    bound = 2e-5 * (w + w.mean())
    for got in (a, other[1]):
        assert (np.linalg.norm(got[:, :3] - ref, axis=1) <= bound).all()
    dv = 2 * bound * np.abs(pos[:, 3]) * DT + 1e-6 * (np.abs(one[1][:, :3]).max(axis=1) + 1e-3)
    assert (np.abs(one[1][:, :3] - other[2][1][:, :3]).max(axis=1) <= dv).all()
    assert one[0][:, 3].tobytes() == pos[:, 3].tobytes() and one[1][:, 3].tobytes() == vel[:, 3].tobytes()


@pytest.mark.parametrize("n,nranks", [(5, 2), (3001, 4), (9001, 3), (24576, 2)])
def test_direct_shards(cuda, n, nranks):
    p, v = ics.plummer(n, seed=n)
    pos, vel = ics.f32(p), ics.f32(v)
    kw = dict(kick="physical", eps2=EPS2, damping=1.0, dt=DT)
    got_p, got_v, _ = run_shards(n, nranks, 3, "f32", "fast", pos, vel, **kw)
    with NBodySystem(n, "f32", "fast", **kw) as s:
        s.set_state(pos, vel)
        s.step(3)
        want_p, want_v = s.get_state()
    assert got_p.tobytes() == want_p.tobytes() and got_v.tobytes() == want_v.tobytes()
