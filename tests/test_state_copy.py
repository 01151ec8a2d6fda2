"""nb_set_state / nb_get_state with NB_DEVICE: the state arrives unchanged
whatever kind of pointer it is (aligned and unaligned device memory, pinned and
pageable host memory, the context's own buffers), for float and double, and the
calls can be captured into a graph."""
import ctypes as C

import numpy as np
import pytest

from utc_gb300 import _native as N
from utc_gb300.nbody import NBodySystem, current_stream_handle

pytestmark = pytest.mark.gpu


def bodies(n, dtype, seed):
    r = np.random.default_rng(seed)
    return r.uniform(-1, 1, (n, 4)).astype(dtype), r.uniform(-1, 1, (n, 4)).astype(dtype)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 70001])
@pytest.mark.parametrize("kind", ["device", "offset", "pinned", "pageable", "own"])
def test_round_trip(cuda, n, prec, kind):
    import torch

    dtype = np.float32 if prec == "f32" else np.float64
    p, v = bodies(n, dtype, n)
    with NBodySystem(n, prec, "exact") as s:

        def buffer(a):
            if kind == "offset":  # one value past an aligned address
                t = torch.empty(4 * n + 1, dtype=torch.from_numpy(a).dtype, device="cuda")[1:].view(n, 4)
            elif kind in ("pinned", "pageable"):
                t = torch.empty((n, 4), dtype=torch.from_numpy(a).dtype, pin_memory=kind == "pinned")
            else:
                t = torch.empty((n, 4), dtype=torch.from_numpy(a).dtype, device="cuda")
            t.copy_(torch.from_numpy(a))
            return t

        a, b = buffer(p), buffer(v)
        st = C.c_void_p(current_stream_handle())
        assert s.lib.nb_set_state(s.handle, a.data_ptr(), b.data_ptr(), N.NB_DEVICE, st) == N.NB_OK
        if kind == "own":  # the current buffers loaded again
            q0, q1 = s.state_ptrs()
            assert s.lib.nb_set_state(s.handle, q0, q1, N.NB_DEVICE, st) == N.NB_OK
        torch.cuda.synchronize()
        gp, gv = s.get_state()
        assert gp.tobytes() == p.tobytes() and gv.tobytes() == v.tobytes()
        c, d = torch.zeros_like(a), torch.zeros_like(b)
        if kind == "offset":
            c, d = buffer(np.zeros_like(p)), buffer(np.zeros_like(v))
        assert s.lib.nb_get_state(s.handle, c.data_ptr(), d.data_ptr(), N.NB_DEVICE, st) == N.NB_OK
        torch.cuda.synchronize()
        assert c.cpu().numpy().tobytes() == p.tobytes() and d.cpu().numpy().tobytes() == v.tobytes()
        # one of the two alone, and crossed destinations (copied in order)
        e = torch.zeros_like(c)
        assert s.lib.nb_get_state(s.handle, None, e.data_ptr(), N.NB_DEVICE, st) == N.NB_OK
        assert s.lib.nb_get_state(s.handle, c.data_ptr(), c.data_ptr(), N.NB_DEVICE, st) == N.NB_OK
        torch.cuda.synchronize()
        assert e.cpu().numpy().tobytes() == v.tobytes() and c.cpu().numpy().tobytes() == v.tobytes()


def test_captured_state_calls(cuda):
    """set_state, a step and get_state_device in a graph that torch captures
    (global mode), replayed on new inputs in the same buffers."""
    import torch

    n = 1024
    p, v = (torch.from_numpy(x).cuda() for x in bodies(n, np.float32, 1))
    p2, v2 = (torch.from_numpy(x).cuda() for x in bodies(n, np.float32, 2))
    p[:, 3] = p2[:, 3] = 1e-3
    out = [torch.empty_like(p) for _ in range(2)]
    with NBodySystem(n, "f32", "sym", kick="physical", eps2=1e-2, dt=1e-3, damping=1.0) as s:
        want = []
        for a, b in ((p, v), (p2, v2)):
            s.set_state(a, b)
            s.step(2)
            s.get_state_device(*out)
            want.append([t.clone() for t in out])
        a, b = p.clone(), v.clone()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            s.set_state(a, b)
            s.step(2)
            s.get_state_device(*out)
        for (x, y), w in zip(((p, v), (p2, v2)), want):
            a.copy_(x)
            b.copy_(y)
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(out[0], w[0]) and torch.equal(out[1], w[1])
