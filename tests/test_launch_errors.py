"""A launch that fails is reported once: the call returns NB_ERR_CUDA, and calls on
other contexts and streams afterwards succeed.  The failure is made on the host: a
capture that a stream synchronisation has invalidated takes no more launches."""
import ctypes as C

import numpy as np
import pytest

from utc_gb300 import _native as N
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem, current_stream_handle

pytestmark = pytest.mark.gpu

THREAD_LOCAL = 1  # CU_STREAM_CAPTURE_MODE_THREAD_LOCAL


@pytest.mark.parametrize("prec,algo,n", [("f32", "sym", 300), ("f32", "sym", 9001), ("f32", "fast", 300), ("f64", "sym", 500),
                                         ("f64", "sym", 7000)])
def test_a_failed_launch_is_reported_once(cuda, prec, algo, n):
    import torch

    cu = C.CDLL("libcuda.so.1")
    cu.cuStreamBeginCapture_v2.argtypes = [C.c_void_p, C.c_int]
    cu.cuStreamSynchronize.argtypes = [C.c_void_p]
    cu.cuStreamEndCapture.argtypes = [C.c_void_p, C.POINTER(C.c_void_p)]
    dtype = np.float32 if prec == "f32" else np.float64
    p, v = (a.astype(dtype) for a in ics.uniform_cube(n, seed=n))
    q, w = (ics.f32(a) for a in ics.uniform_cube(64, seed=1))
    stream = torch.cuda.Stream()
    st = C.c_void_p(stream.cuda_stream)
    here = C.c_void_p(current_stream_handle())
    with NBodySystem(n, prec, algo) as s, NBodySystem(n, prec, algo) as t, NBodySystem(64, "f32", "exact") as other:
        for x in (s, t):
            x.set_state(p, v)
        other.set_state(q, w)
        torch.cuda.synchronize()
        assert cu.cuStreamBeginCapture_v2(st, THREAD_LOCAL) == 0
        assert cu.cuStreamSynchronize(st) != 0  # invalidates the capture
        failed = s.lib.nb_step(s.handle, 1, st)
        graph = C.c_void_p()
        assert cu.cuStreamEndCapture(st, C.byref(graph)) != 0 and not graph.value
        assert failed == N.NB_ERR_CUDA
        # plain launches check the error that the runtime holds
        assert other.lib.nb_step(other.handle, 1, here) == N.NB_OK, N.lib().nb_last_error()
        # the context is as before the failed call
        for x in (s, t):
            x.step(2)
        a, b = s.get_state(), t.get_state()
    assert a[0].tobytes() == b[0].tobytes() and a[1].tobytes() == b[1].tobytes()
