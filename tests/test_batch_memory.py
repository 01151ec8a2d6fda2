"""A batch of the automatic shape (12 targets per lane) whose source-side array does
not fit the free memory is planned with 16, whose array is 3/4 as large."""
import numpy as np
import pytest

from utc_gb300 import _native as N
from utc_gb300 import ics
from utc_gb300.nbody import NBodyBatch

pytestmark = pytest.mark.gpu

MIB = 1 << 20
SIZES = [150000]  # arrays n^2 / (2 rb) of 16 bytes: 446 MiB with 12 targets (rb = 384), 334 MiB with 16


def test_the_smaller_array_is_taken_where_it_alone_fits(cuda):
    import torch

    p, v = ics.plummer(SIZES[0], seed=2)
    pos, vel = ics.f32(p), ics.f32(v)
    kw = dict(kick="physical", eps2=np.float32(1e-4), damping=1.0, dt=np.float32(1e-4))
    with NBodyBatch(SIZES, **kw) as b:
        assert b.plan_info()["bodies_per_lane"] == 12
    with NBodyBatch(SIZES, warps_per_cta=1, bodies_per_lane=16, **kw) as b:
        b.set_state(pos, vel)
        b.step(2)
        want = b.get_state()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty((torch.cuda.mem_get_info()[0] - 430 * MIB,), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(N.NbError) as e:
            NBodyBatch(SIZES, warps_per_cta=1, bodies_per_lane=12, **kw)
        assert e.value.status == N.NB_ERR_OOM  # an explicit shape is what was asked for
        with NBodyBatch(SIZES, **kw) as b:
            assert b.plan_info()["bodies_per_lane"] == 16
            b.set_state(pos, vel)
            b.step(2)
            got = b.get_state()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()
