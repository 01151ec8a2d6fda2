"""The one-launch step of small FP64 systems in float-float arithmetic
(utc_gb300/csrc/nb_symff.cu): at the edges of its tiles (two bodies a CTA, 128
threads, the largest size that it takes and the first that it does not)
accelerations within 1e-13 (|a| + mean|a|) of the FP64 oracle, a hundred times
what float-float rounding leaves, and one step's state within that times dt
plus two roundings; graph replay, launches, a second context and a batch's
per-system steps give the same bits; the energy pass is another kernel's."""
import numpy as np
import pytest

import oracle
from utc_gb300 import ics
from utc_gb300.nbody import NBodyBatch, NBodySystem

pytestmark = pytest.mark.gpu

EPS2, DT, DAMP = 2.0 ** -10, 2.0 ** -10, 0.999


@pytest.mark.parametrize("kick", ["physical", "reference"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 64, 65, 127, 128, 129, 255, 257, 1000, 2047, 2399, 2400, 2401])
def test_small_ff_step_vs_oracle(cuda, n, kick):
    pos, vel = ics.uniform_cube(n, seed=n)
    args = dict(kick=kick, eps2=EPS2, damping=DAMP, dt=DT)
    outs = []
    for _ in range(2):
        with NBodySystem(n, "f64", "sym", **args) as s:
            assert s.launches_per_step() == (2 if n <= 2400 else 3)
            s.set_state(pos, vel)
            a = s.accel()
            s.step(1)
            one = s.get_state()
            s.step(34)  # 2 replayed graphs and 2 launches
            outs.append((a, one, s.get_state(), s.energy()))
    with NBodySystem(n, "f64", "sym", **args) as s:
        s.set_state(pos, vel)
        for _ in range(35):
            s.step(1)
        single = s.get_state()
    ref = oracle.accel(pos, EPS2)[:, :3]
    d, w = np.linalg.norm(outs[0][0][:, :3] - ref, axis=1), np.linalg.norm(ref, axis=1)
    bound = 1e-13 * (w + w.mean())
    assert (d <= bound).all()
    k = pos[:, 3] if kick == "reference" else np.ones(n)
    km = oracle.KICK_REFERENCE if kick == "reference" else oracle.KICK_PHYSICAL
    want, wv = oracle.step(pos, vel, EPS2, DAMP, DT, 1, kick_mode=km)
    gp, gv = outs[0][1]
    dv = bound * np.abs(k) * DT + 2 ** -51 * np.abs(wv[:, :3]).max(axis=1)
    assert (np.abs(gv[:, :3] - wv[:, :3]).max(axis=1) <= dv).all()
    assert (np.abs(gp[:, :3] - want[:, :3]).max(axis=1) <= dv * DT + 2 ** -51 * np.abs(want[:, :3]).max(axis=1)).all()
    assert gp[:, 3].tobytes() == pos[:, 3].tobytes() and gv[:, 3].tobytes() == vel[:, 3].tobytes()
    for c in range(2):
        assert outs[0][2][c].tobytes() == outs[1][2][c].tobytes() == single[c].tobytes()
    assert np.array_equal(outs[0][3], outs[1][3])


def test_small_ff_in_a_batch(cuda):
    """A batch's per-system steps take the same path for its small systems."""
    sizes = [7, 2401, 600, 2400]
    states = [ics.uniform_cube(n, seed=n) for n in sizes]
    with NBodyBatch(sizes, precision="f64", kick="physical", eps2=EPS2, damping=DAMP, dt=DT) as b:
        b.set_state(np.concatenate([p for p, _ in states]), np.concatenate([v for _, v in states]))
        b.step_per_system(2)
        bp, bv = b.get_state()
    bp, bv = (np.concatenate(x) if isinstance(x, (list, tuple)) else x for x in (bp, bv))
    o = 0
    for n, (p, v) in zip(sizes, states):
        with NBodySystem(n, "f64", "sym", kick="physical", eps2=EPS2, damping=DAMP, dt=DT) as s:
            s.set_state(p, v)
            s.step(2)
            gp, gv = s.get_state()
        assert bp[o:o + n].tobytes() == gp.tobytes() and bv[o:o + n].tobytes() == gv.tobytes()
        o += n
