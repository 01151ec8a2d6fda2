"""The forward pass of the adjoint keeps every state where they come to at most
1 GiB and checkpoints beyond (nb_adj_forward): the gradients of a trajectory
just above that size (checkpoints, recomputed segments) are, bit for bit, those
of its two halves (each of them kept whole) chained by hand."""
import numpy as np
import pytest

from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo,kick,n", [("sym", "physical", 9001), ("sym", "reference", 8000), ("fast", "physical", 9001),
                                         ("fast", "reference", 4097)])
def test_checkpointed_equals_kept_halves(cuda, algo, kick, n):
    import torch

    per = 32 if kick == "reference" else 16
    half = (2 ** 30 // (per * n) + 2) // 2
    steps = 2 * half
    assert steps * per * n > 2 ** 30 > (half + 1) * per * n
    p, v = ics.uniform_cube(n, seed=3)
    pos, vel = torch.tensor(ics.f32(p), device="cuda"), torch.tensor(ics.f32(v), device="cuda")
    torch.manual_seed(1)
    gx, gv = torch.randn((n, 4), device="cuda"), torch.randn((n, 4), device="cuda")
    gx[:, 3] = gv[:, 3] = 0
    kw = dict(kick=kick, eps2=np.float32(1e-2), damping=1.0, dt=np.float32(1e-5))
    x1, v1, xt, vt = (torch.empty_like(pos) for _ in range(4))
    with NBodySystem(n, "f32", algo, **kw) as s:
        s.set_state(pos, vel)
        s.adj_forward(half, 100)
        s.get_state_device(x1, v1)
        s.adj_forward(half, 100)
        s.get_state_device(xt, vt)
        bx, bv, bm = s.adj_backward(gx, gv)
        s.set_state(pos, vel)
        s.adj_forward(half, 100)
        want = s.adj_backward(bx, bv)
    with NBodySystem(n, "f32", algo, **kw) as s:
        s.set_state(pos, vel)
        s.adj_forward(steps, 500)
        x2, v2 = torch.empty_like(pos), torch.empty_like(pos)
        s.get_state_device(x2, v2)
        got = s.adj_backward(gx, gv)
        again = s.adj_backward(gx, gv)
    assert torch.equal(x2, xt) and torch.equal(v2, vt)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    m = (want[2] + bm).double()  # one running sum against two: rounding only
    assert float((got[2].double() - m).norm()) <= 1e-4 * float(m.norm())
    for a, b in zip(got, again):
        assert torch.equal(a, b)
