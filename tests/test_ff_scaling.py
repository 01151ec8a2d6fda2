"""The scaling and splitting that the float-float step (NB_F64 with
NB_ALGO_SYM) starts with, at the edges of its two forms (blocks of 64 bodies,
256 bodies a pass, one launch up to 6144 bodies and three above): coordinates
times 2^k and masses times 2^j give accelerations times 2^(j - 2 k), bit for
bit, since the scale is an exact power of two and everything after the split
runs in scaled units; and the accelerations are the FP64 oracle's to 1e-13
(|a| + mean|a|), a hundred times what float-float rounding leaves."""
import numpy as np
import pytest

import oracle
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

pytestmark = pytest.mark.gpu

EPS2 = 2.0 ** -10


def _accel(pos, eps2):
    with NBodySystem(len(pos), "f64", "sym", kick="physical", eps2=eps2, dt=2.0 ** -10) as s:
        s.set_state(pos, np.zeros_like(pos))
        return s.accel()[:, :3].copy()


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 257, 2047, 2049, 4097, 6143, 6144, 6145, 8193])
def test_scales_are_exact(cuda, n):
    pos, _ = ics.uniform_cube(n, seed=n)
    pos[:, 3] = np.random.default_rng(n).uniform(0.1, 3.0, n)
    base = _accel(pos, EPS2)
    ref = oracle.accel(pos, EPS2)
    d, w = np.linalg.norm(base - ref[:, :3], axis=1), np.linalg.norm(ref[:, :3], axis=1)
    assert (d <= 1e-13 * (w + w.mean())).all()
    for k, j in ((400, -100), (-400, 100), (0, 900), (150, -700), (-1, -1)):
        q = pos.copy()
        q[:, :3] = np.ldexp(q[:, :3], k)
        q[:, 3] = np.ldexp(q[:, 3], j)
        got = _accel(q, float(np.ldexp(EPS2, 2 * k)))
        assert got.tobytes() == np.ldexp(base, j - 2 * k).tobytes(), (k, j)


def test_scale_sees_every_body(cuda):
    """The largest coordinate and the largest mass in the first, a middle and
    the last body, by themselves."""
    n = 3001
    for at in (0, 1, 1500, n - 1):
        pos, _ = ics.uniform_cube(n, seed=3)
        pos[at, :3] = (1e4, -3e4, 2e4)
        pos[(at + 7) % n, 3] = 5e3
        ref = oracle.accel(pos, EPS2)
        d = np.linalg.norm(_accel(pos, EPS2) - ref[:, :3], axis=1)
        w = np.linalg.norm(ref[:, :3], axis=1)
        assert (d <= 1e-13 * (w + w.mean())).all()
