"""Plummer bodies as floats are formed in float-float arithmetic where the scale
radius and the speed scale lie within 2^40 of one, in FP64 beyond: on either side
of both ends positions in units of a and velocities in units of sqrt(G M / a)
are the same draws, to a few roundings of a float (each side within 2 ulp of the
exact value, the common shift of the centre included: 4 * 2^-23)."""
import numpy as np
import pytest

from utc_gb300.nbody import gpu_initial_conditions

pytestmark = pytest.mark.gpu


def _units(n, a, gm):
    pos, vel = (x.cpu().numpy().astype(np.float64) for x in
                gpu_initial_conditions("plummer", n, seed=7, a=a, G=1.0, M=gm, precision="f32"))
    assert np.isfinite(pos).all() and np.isfinite(vel).all()
    assert np.allclose(pos[:, 3], gm / n, rtol=1e-6)
    return pos[:, :3] / a, vel[:, :3] / np.sqrt(gm / a)


@pytest.mark.parametrize("n", [1, 100, 2049])
def test_plummer_units(cuda, n):
    base = _units(n, 1.0, 1.0)
    for a, gm in ((2.0 ** 40, 2.0 ** 40), (2.0 ** 41, 2.0 ** 41), (2.0 ** -40, 2.0 ** -40), (2.0 ** -41, 2.0 ** -41),
                  (1.0, 2.0 ** 78), (1.0, 2.0 ** 82), (1.0, 2.0 ** -80), (1.0, 2.0 ** -82), (2.0 ** 50, 1.0)):
        for got, want in zip(_units(n, a, gm), base):
            w = np.abs(want).max(axis=1, keepdims=True)
            assert (np.abs(got - want) <= 2.0 ** -21 * (w + w.mean())).all(), (a, gm)
