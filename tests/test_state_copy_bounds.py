"""nb_set_state / nb_get_state with NB_DEVICE refuse a buffer that ends before the
state does, as a copy does (NB_ERR_CUDA), and take one that ends exactly with it.

The short buffers are the first of a run of contiguous 512-byte allocations that
are all this test's own: a call that did not refuse would stay inside them."""
import ctypes as C

import numpy as np
import pytest

from utc_gb300 import _native as N
from utc_gb300.nbody import NBodySystem, current_stream_handle

pytestmark = pytest.mark.gpu

SMALL, BLOCKS = 512, 64


@pytest.fixture
def blocks(cuda):
    """Addresses of BLOCKS contiguous 512-byte allocations."""
    import torch

    torch.zeros(1, device="cuda")
    cu = C.CDLL("libcuda.so.1")
    cu.cuMemAlloc_v2.argtypes = [C.POINTER(C.c_uint64), C.c_size_t]
    cu.cuMemFree_v2.argtypes = [C.c_uint64]
    got = []
    try:
        for _ in range(BLOCKS):
            d = C.c_uint64()
            assert cu.cuMemAlloc_v2(C.byref(d), SMALL) == 0
            got.append(d.value)
        got.sort()
        runs = [k for k in range(BLOCKS - 16) if got[k + 16] - got[k] == 16 * SMALL]
        if not runs:
            pytest.skip("the allocations are not contiguous")
        yield got[runs[0]:runs[0] + 16]
    finally:
        torch.cuda.synchronize()
        for d in got:
            cu.cuMemFree_v2(d)


@pytest.mark.parametrize("prec,n", [("f32", 128), ("f64", 64), ("f32", 33)])
def test_short_buffers_are_refused(blocks, prec, n):
    import torch

    dtype = np.float32 if prec == "f32" else np.float64
    sb = 4 * n * np.dtype(dtype).itemsize
    assert SMALL < sb <= 4 * SMALL
    r = np.random.default_rng(n)
    p, v = r.uniform(-1, 1, (n, 4)).astype(dtype), r.uniform(-1, 1, (n, 4)).astype(dtype)
    st = C.c_void_p(current_stream_handle())
    with NBodySystem(n, prec, "exact") as s:
        s.set_state(torch.tensor(p, device="cuda"), torch.tensor(v, device="cuda"))
        short, other = blocks[0], blocks[8]
        full = torch.zeros((n, 4), dtype=torch.from_numpy(p).dtype, device="cuda")
        for a, b in ((short, full.data_ptr()), (full.data_ptr(), short), (short, other)):
            assert s.lib.nb_get_state(s.handle, a, b, N.NB_DEVICE, st) == N.NB_ERR_CUDA
        torch.cuda.synchronize()
        gp, gv = s.get_state()
        assert gp.tobytes() == p.tobytes() and gv.tobytes() == v.tobytes()
        for a, b in ((short, full.data_ptr()), (full.data_ptr(), short), (short, other)):
            assert s.lib.nb_set_state(s.handle, a, b, N.NB_DEVICE, st) == N.NB_ERR_CUDA
        torch.cuda.synchronize()


@pytest.mark.parametrize("n,short", [(32, 0), (31, 16)])
def test_buffers_that_end_with_the_state_are_taken(blocks, n, short):
    """32 bodies fill a block; 31 end with it from its 16th byte on."""
    r = np.random.default_rng(n)
    p, v = r.uniform(-1, 1, (n, 4)).astype(np.float32), r.uniform(-1, 1, (n, 4)).astype(np.float32)
    st = C.c_void_p(current_stream_handle())
    with NBodySystem(n, "f32", "exact") as s, NBodySystem(n, "f32", "exact") as t:
        s.set_state(p, v)
        a, b = blocks[0] + short, blocks[5] + short
        assert s.lib.nb_get_state(s.handle, a, b, N.NB_DEVICE, st) == N.NB_OK
        assert t.lib.nb_set_state(t.handle, a, b, N.NB_DEVICE, st) == N.NB_OK
        gp, gv = t.get_state()
    assert gp.tobytes() == p.tobytes() and gv.tobytes() == v.tobytes()
