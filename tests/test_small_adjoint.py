"""The one-launch reverse step of small systems (utc_gb300/csrc/nb_adjoint.cu) at
the edges of its tiles (four bodies a CTA, 128 threads, the largest size that
it takes and the first that it does not): gradients within 1e-4 in norm of the
FP64 oracle, as of the symmetric kernels; odd step counts (both halves of the
alternating buffer) and a second backward pass give the same bits."""
import numpy as np
import pytest

import oracle
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kick", ["physical", "reference"])
@pytest.mark.parametrize("n,steps,every", [(1, 3, 2), (2, 4, 4), (3, 5, 2), (4, 1, 1), (5, 6, 3), (127, 5, 2), (128, 4, 3),
                                           (129, 3, 1), (1001, 3, 2), (6999, 2, 1), (7000, 1, 1), (7001, 2, 2)])
def test_small_reverse_steps(cuda, n, steps, every, kick):
    import torch

    p, v = ics.uniform_cube(n, seed=n)
    if kick == "reference":
        p[:, 3] *= 100
    pos, vel = ics.f32(p), ics.f32(v)
    y = ics.gaussian_targets(n, seed=n + 1)
    eps2, dt = float(np.float32(1e-2)), float(np.float32(1e-3))
    with NBodySystem(n, "f32", "sym", kick=kick, eps2=eps2, damping=1.0, dt=dt) as s:
        s.set_state(pos, vel)
        s.adj_forward(steps, every)
        pT, _ = s.get_state()
        gx = torch.zeros((n, 4), device="cuda")
        gx[:, :3] = torch.tensor(2 * (pT[:, :3].astype(np.float64) - y), dtype=torch.float32, device="cuda")
        first = [t.cpu().numpy() for t in s.adj_backward(gx)]
        second = [t.cpu().numpy() for t in s.adj_backward(gx)]
    for a, b in zip(first, second):
        assert a.tobytes() == b.tobytes()
    km = oracle.KICK_REFERENCE if kick == "reference" else oracle.KICK_PHYSICAL
    _, rx, rv, rm = oracle.adjoint(pos.astype(np.float64), vel.astype(np.float64), y, eps2, 1.0, dt, steps, kick_mode=km)
    for got, want in ((first[0][:, :3], rx), (first[1][:, :3], rv), (first[2], rm)):
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want) + 1e-12
