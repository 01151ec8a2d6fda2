"""Directed FP32 pair terms over the float range.  The weight m / d^3 is formed
as (m / d) / d^2: 1 / d^3 by itself is subnormal from d = 4.4e12 on and
overflows below 1.4e-13, which with a softening that small makes the self
pair's 0 * inf NaN.  Bodies of 1e30 kg at 1e13 to 1e18 m, and bodies of 1e-10
with eps2 = 1e-30, on every path that evaluates pairs from the target's side
only: directed contexts on either side of 24576 bodies and their shards, the
allocation-free step, symmetric contexts of up to 9000 bodies and of one row
block, batches of systems of one row block.

Bound: 2e-5 (|a| + mean|a|) per body against the FP64 oracle, as the same cube
is held to at unit scale (tests/test_direct.py): every product of the weight is
a normal float at these scales, so its relative error is the one at unit scale."""
import numpy as np
import pytest

import oracle
from test_shard_gpu import run_shards
from utc_gb300 import ics
from utc_gb300.nbody import NBodyBatch, NBodySystem

pytestmark = pytest.mark.gpu

# (length, mass, softening squared)
SCALES = [(1e13, 1e30, 1e23), (1e14, 1e30, 1e25), (1e15, 1e30, 1e27), (1e18, 1e30, 1e33), (1.0, 1e-10, 1e-30)]


def bodies(n, length, mass, seed):
    p, v = ics.uniform_cube(n, seed=seed)
    p[:, :3] *= length
    p[:, 3] *= mass
    v[:, :3] = 0.0
    return ics.f32(p), ics.f32(v)


def check(a, pos, eps2):
    ref = oracle.accel(pos.astype(np.float64), eps2)[:, :3]
    w = np.linalg.norm(ref, axis=1)
    assert np.isfinite(a).all()
    assert (np.linalg.norm(a[:, :3].astype(np.float64) - ref, axis=1) <= 2e-5 * (w + w.mean())).all()


# explicit shapes that are not the automatic one: the symmetric kernel itself
@pytest.mark.parametrize("algo,n,kw", [("fast", 300, {}), ("fast", 12000, {}), ("fast", 24577, {}), ("sym", 100, {}),
                                       ("sym", 3000, {}), ("sym", 500, dict(block=32, bpt=16)),
                                       ("sym", 2500, dict(block=128, bpt=20))])
@pytest.mark.parametrize("length,mass,eps2", SCALES)
def test_single_system(cuda, algo, n, kw, length, mass, eps2):
    eps2 = float(np.float32(eps2))
    pos, vel = bodies(n, length, mass, n)
    with NBodySystem(n, "f32", algo, kick="physical", eps2=eps2, damping=1.0, dt=1.0, **kw) as s:
        s.set_state(pos, vel)
        check(s.accel(), pos, eps2)


def test_small_softening_beyond_one_row_block(cuda):
    """Symmetric contexts of many row blocks: the own-row chunks hold the self
    pairs, the others' inverse cubes stay finite at these distances."""
    n, eps2 = 10000, float(np.float32(1e-30))
    pos, vel = bodies(n, 1.0, 1e-10, 5)
    for kw in ({}, dict(bands=3)):
        with NBodySystem(n, "f32", "sym", kick="physical", eps2=eps2, damping=1.0, dt=1.0, **kw) as s:
            s.set_state(pos, vel)
            check(s.accel(), pos, eps2)


@pytest.mark.parametrize("length,mass,eps2", SCALES)
def test_batch_of_one_row_block_systems(cuda, length, mass, eps2):
    """One step of dt = 1 from rest: the velocities are the accelerations."""
    eps2 = float(np.float32(eps2))
    sizes = [1, 33, 250, 384]
    parts = [bodies(k, length, mass, 7 + k) for k in sizes]
    pos, vel = (np.concatenate([p[q] for p in parts]) for q in (0, 1))
    with NBodyBatch(sizes, kick="physical", eps2=eps2, damping=1.0, dt=1.0, G=1.0) as b:
        b.set_state(pos, vel)
        b.step(1)
        _, got = b.get_state()
    o = np.concatenate([[0], np.cumsum(sizes)])
    for s, k in enumerate(sizes):
        if k > 1:
            check(got[o[s]:o[s + 1]], pos[o[s]:o[s + 1]], eps2)
        else:
            assert (got[o[s], :3] == 0).all()


def test_shards_and_allocation_free_step(cuda):
    import ctypes as C

    import torch

    from utc_gb300 import _native as N
    from utc_gb300.nbody import current_stream_handle

    n, eps2 = 9000, float(np.float32(1e33))
    pos, vel = bodies(n, 1e18, 1e30, 3)
    kw = dict(kick="physical", eps2=eps2, damping=1.0, dt=1.0)
    _, got, _ = run_shards(n, 3, 1, "f32", "fast", pos, vel, **kw)
    check(got, pos, eps2)
    p, v = torch.tensor(pos, device="cuda"), torch.tensor(vel, device="cuda")
    out = torch.empty_like(p)
    N.check(N.lib().nb_step_f32_noalloc(C.c_void_p(p.data_ptr()), C.c_void_p(out.data_ptr()), C.c_void_p(v.data_ptr()), n,
                                        eps2, 1.0, 1.0, N.NB_KICK_PHYSICAL, 1.0, C.c_void_p(current_stream_handle())))
    torch.cuda.synchronize()
    check(v.cpu().numpy(), pos, eps2)
