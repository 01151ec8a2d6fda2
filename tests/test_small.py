"""The one-launch step of small FP32 symmetric systems (utc_gb300/csrc/
nb_small.cu): at sizes around its tile edges (targets per CTA, 128 threads, the
changes of tile, the largest size that it takes and the first that it does
not) accelerations within 2e-5 (|a| + mean|a|) and one step's positions within
1e-5 (|x| + 0.1) of the FP64 oracle, the tolerances of the symmetric kernels;
graph replay, launches and a second context give the same bits."""
import numpy as np
import pytest

import oracle
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

pytestmark = pytest.mark.gpu

EPS2, DT = np.float32(1e-3), np.float32(1e-3)


@pytest.mark.parametrize("kick", ["physical", "reference"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 127, 128, 129, 511, 1023, 1999, 2000, 2001, 2999, 3001, 8999, 9000,
                               9001])
def test_small_step_vs_oracle(cuda, n, kick):
    p, v = ics.uniform_cube(n, seed=n)
    pos, vel = ics.f32(p), ics.f32(v)
    outs = []
    for _ in range(2):
        with NBodySystem(n, "f32", "sym", kick=kick, eps2=EPS2, damping=np.float32(0.999), dt=DT) as s:
            assert s.launches_per_step() == (1 if n <= 9000 else 2)
            s.set_state(pos, vel)
            a = s.accel()
            s.step(1)
            one = s.get_state()
            s.step(34)  # 2 replayed graphs and 2 launches
            outs.append((a, one, s.get_state()))
    with NBodySystem(n, "f32", "sym", kick=kick, eps2=EPS2, damping=np.float32(0.999), dt=DT) as s:
        s.set_state(pos, vel)
        for _ in range(35):
            s.step(1)
        single = s.get_state()
    ref = oracle.accel(pos.astype(np.float64), float(EPS2))
    d, w = np.linalg.norm(outs[0][0] - ref, axis=1), np.linalg.norm(ref, axis=1)
    assert (d <= 2e-5 * (w + w.mean())).all()
    km = oracle.KICK_REFERENCE if kick == "reference" else oracle.KICK_PHYSICAL
    want, wv = oracle.step(pos.astype(np.float64), vel.astype(np.float64), float(EPS2), float(np.float32(0.999)),
                           float(DT), 1, kick_mode=km)
    (gp, gv) = outs[0][1]
    assert np.abs(gp[:, :3] - want[:, :3]).max() <= 1e-5 * (np.abs(want[:, :3]).max() + 0.1)
    assert np.abs(gv[:, :3] - wv[:, :3]).max() <= 1e-5 * (np.abs(wv[:, :3]).max() + 0.1)
    assert gp[:, 3].tobytes() == pos[:, 3].tobytes() and gv[:, 3].tobytes() == vel[:, 3].tobytes()
    for k in range(2):
        assert outs[0][2][k].tobytes() == outs[1][2][k].tobytes() == single[k].tobytes()


def test_small_step_shape_given_or_not(cuda):
    """The automatic shape, given explicitly, is the same plan; another shape
    is the symmetric kernels', within their tolerance."""
    n = 1500
    p, v = ics.plummer(n, seed=5)
    pos, vel = ics.f32(p), ics.f32(v)
    got = []
    for kw in ({}, {"block": 32, "bpt": 4}, {"block": 32, "bpt": 16}, {"bands": 2}, {"source_side": "fixed"}):
        with NBodySystem(n, "f32", "sym", kick="physical", eps2=EPS2, damping=1.0, dt=DT, **kw) as s:
            s.set_state(pos, vel)
            s.step(3)
            got.append((s.launches_per_step(), s.get_state()[0]))
    assert [g[0] for g in got][:3] == [1, 1, 2] and got[3][0] > 2 and got[4][0] == 2
    assert got[0][1].tobytes() == got[1][1].tobytes()
    for _, q in got[2:]:
        assert np.abs(q - got[0][1]).max() <= 1e-5
