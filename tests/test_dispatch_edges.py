"""The kernels above the small systems' sizes, at the edge sizes that the default
shapes leave to the small kernels: the stream-K directed kernel by an explicit
shape, its shards at sizes with fewer target blocks than ranks, and the symmetric
kernels by explicit shapes and at odd sizes just above 9000 (float) and 2400
(double).  Tolerances are those of the kernels' own tests (2e-5 and 1e-13 of
|a| + mean|a| against the FP64 oracle)."""
import ctypes as C

import numpy as np
import pytest

import oracle
import test_shard_gpu
from utc_gb300 import _native as N
from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem
from utc_gb300.shard import block_split

pytestmark = pytest.mark.gpu

BLOCK, BPT = 256, 4  # target blocks of 1024; automatic at none of these sizes
EPS2, DT = float(np.float32(1e-3)), float(np.float32(1e-3))


class ShapedShard(test_shard_gpu.Shard):
    def __init__(self, n, rank, nranks, precision, algo, **kw):
        self.lib = N.lib()
        p = N.NbParams()
        self.lib.nb_params_default(C.byref(p))
        p.n, p.precision, p.algo, p.kick = n, N.NB_F32, N.NB_ALGO_FAST, N.NB_KICK_PHYSICAL
        p.block, p.bpt = BLOCK, BPT
        p.eps2, p.damping, p.dt = kw["eps2"], kw["damping"], kw["dt"]
        self.h = C.c_void_p()
        N.check(self.lib.nb_create_shard(C.byref(p), rank, nranks, C.byref(self.h)), "nb_create_shard")
        info = (C.c_int * 4)()
        N.check(self.lib.nb_shard_info(self.h, info), "nb_shard_info")
        self.first, self.count, self.n = info[0], info[1], n
        self.dtype, self.typestr = np.float32, "<f4"


def close_to_oracle(a, pos, eps2, tol):
    ref = oracle.accel(pos.astype(np.float64), eps2)[:, :3]
    w = np.linalg.norm(ref, axis=1)
    assert (np.linalg.norm(a[:, :3] - ref, axis=1) <= tol * (w + w.mean())).all()


@pytest.mark.parametrize("n,nranks", [(1, 2), (2, 3), (5, 8), (1001, 3), (1024, 2), (1025, 2), (1025, 3), (5000, 4), (9001, 7),
                                      (24576, 3)])
def test_stream_k_shards(cuda, monkeypatch, n, nranks):
    p, v = ics.plummer(n, seed=n)
    pos, vel = ics.f32(p), ics.f32(v)
    kw = dict(kick="physical", eps2=EPS2, damping=1.0, dt=DT)
    monkeypatch.setattr(test_shard_gpu, "Shard", ShapedShard)
    got_p, got_v, ranges = test_shard_gpu.run_shards(n, nranks, 3, "f32", "fast", pos, vel, **kw)
    with NBodySystem(n, "f32", "fast", block=BLOCK, bpt=BPT, **kw) as s:
        assert s.plan_info()["tbsize"] == 1024
        s.set_state(pos, vel)
        close_to_oracle(s.accel(), pos, EPS2, 2e-5)
        s.step(3)
        want_p, want_v = s.get_state()
    assert ranges == block_split(n, 1024, nranks) and sum(c for _, c in ranges) == n
    assert got_p.tobytes() == want_p.tobytes() and got_v.tobytes() == want_v.tobytes()


@pytest.mark.parametrize("n,shape", [(n, (32, 16)) for n in (1, 2, 31, 33, 511, 512, 513, 1001, 2500)]
                         + [(n, (128, 20)) for n in (1, 33, 2559, 2560, 2561, 5121)]
                         + [(n, (0, 0)) for n in (9001, 9005, 9215, 9216, 9217, 9249, 10001)])
def test_symmetric_float(cuda, n, shape):
    p, v = ics.uniform_cube(n, seed=n)
    pos, vel = ics.f32(p), ics.f32(v)
    kw = dict(kick="physical", eps2=EPS2, damping=1.0, dt=DT, block=shape[0], bpt=shape[1])
    outs = []
    for steps in ((3,), (1, 1, 1)):
        with NBodySystem(n, "f32", "sym", **kw) as s:
            assert s.launches_per_step() == 2
            s.set_state(pos, vel)
            close_to_oracle(s.accel(), pos, EPS2, 2e-5)
            for k in steps:
                s.step(k)
            outs.append([a.tobytes() for a in s.get_state()])
    assert outs[0] == outs[1]


@pytest.mark.parametrize("n,shape", [(n, (32, 4)) for n in (1, 2, 33, 127, 129, 1001, 2400)]
                         + [(n, (0, 0)) for n in (2401, 2402, 2431, 2432, 2433, 2497)])
def test_symmetric_double(cuda, n, shape):
    pos, vel = ics.uniform_cube(n, seed=n)
    kw = dict(kick="physical", eps2=EPS2, damping=1.0, dt=DT, block=shape[0], bpt=shape[1])
    outs = []
    for steps in ((3,), (1, 1, 1)):
        with NBodySystem(n, "f64", "sym", **kw) as s:
            assert s.launches_per_step() == 3
            s.set_state(pos, vel)
            close_to_oracle(s.accel(), pos, EPS2, 1e-13)
            for k in steps:
                s.step(k)
            outs.append([a.tobytes() for a in s.get_state()])
    assert outs[0] == outs[1]
