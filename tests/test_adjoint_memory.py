"""What nb_adj_forward keeps, and how much memory that takes: all states within
nb_adj_tape_limit and an eighth of the free memory, checkpoints otherwise, never
the buffers of both; the gradients have the same bits either way."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from utc_gb300 import ics
from utc_gb300.nbody import NBodySystem

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
GIB, MIB = 1 << 30, 1 << 20


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("tape") / "adj_tape_probe")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-I", os.path.join(REPO, "include"), "-I",
                    os.path.join(REPO, "utc_gb300", "csrc"), os.path.join(HERE, "adj_tape_probe.cu"), "-o", out],
                   check=True, capture_output=True)
    return lambda *a: subprocess.run([out] + [str(int(x)) for x in a], check=True, capture_output=True,
                                     text=True).stdout.strip() == "1"


@pytest.mark.parametrize("n,steps", [(0, 5), (1, 1), (4096, 16383), (4096, 16384), (4097, 16383), (1 << 26, 1), (1 << 25, 1),
                                     (1 << 30, (1 << 31) - 1), ((1 << 30) - 1, 1 << 30), (1, (1 << 31) - 1)])
@pytest.mark.parametrize("ref", [False, True])
@pytest.mark.parametrize("limit", [0, 1, GIB, 64 * GIB, (1 << 64) - 1])
def test_the_rule_counts_every_byte(fits, n, steps, ref, limit):
    """Python's integers do not wrap: 2^30 bodies x 2^31 states are 2^65 bytes."""
    need = 16 * n * (steps + 1 + (steps if ref else 0))
    assert fits(n, steps, ref, limit) == (n > 0 and need <= limit)


def system(n, algo, **kw):
    if algo == "symfx":
        return NBodySystem(n, "f32", "sym", source_side="fixed", **kw)
    if algo == "symband":
        return NBodySystem(n, "f32", "sym", bands=3, **kw)
    return NBodySystem(n, "f32", algo, **kw)


# small_vjp up to 7000 bodies; symmetric and directed kernels on all sides of it
@pytest.mark.gpu
@pytest.mark.parametrize("algo", ["fast", "sym", "symfx", "symband"])
@pytest.mark.parametrize("kick", ["physical", "reference"])
@pytest.mark.parametrize("n,steps", [(1, 3), (300, 24), (700, 17), (7000, 6), (7001, 6), (9001, 5)])
def test_checkpoints_give_the_bits_of_kept_states(cuda, algo, kick, n, steps):
    import torch

    p, v = ics.uniform_cube(n, seed=n)
    if kick == "reference":
        p[:, 3] *= n
    pos, vel = ics.f32(p), ics.f32(v)
    torch.manual_seed(n)
    gx, gv = torch.randn((n, 4), device="cuda"), torch.randn((n, 4), device="cuda")

    def bits(s, every, limit):
        s.adj_tape_limit(limit)
        s.set_state(pos, vel)
        s.adj_forward(steps, every)
        state = s.get_state()
        first = [t.cpu().numpy().tobytes() for t in s.adj_backward(gx, gv)]
        # the first backward uses the last segment as the forward left it, the
        # second recomputes that one too
        assert [t.cpu().numpy().tobytes() for t in s.adj_backward(gx, gv)] == first
        return [a.tobytes() for a in state] + first

    with system(n, algo, kick=kick, eps2=np.float32(1e-2), damping=0.999, dt=np.float32(1e-3)) as s:
        want = bits(s, 5, GIB)
        for every in (1, 2, 5, steps - 1, steps):
            assert bits(s, every, 0) == want, every
        assert bits(s, 1, GIB) == want
        s.set_state(pos, vel)
        s.step(steps)
        assert [a.tobytes() for a in s.get_state()] == want[:2]


def free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


N, SHORT, LONG = 4096, 8000, 17000  # SHORT: 524 MB of states; LONG: 1.11 GB, beyond the limit


@pytest.mark.gpu
def test_buffers_of_one_kind_of_pass_are_held(cuda):
    """Checkpoints every 200 of LONG steps: 85 + 85 checkpoint arrays and 4 x 200
    segment arrays of 64 KiB, 61 MiB; every 2000: 508 MiB."""
    p, v = ics.plummer(N, seed=1)
    with NBodySystem(N, "f32", "sym", kick="physical", eps2=np.float32(1e-2), damping=1.0, dt=np.float32(1e-6)) as s:
        s.set_state(ics.f32(p), ics.f32(v))
        s.adj_forward(2, 1)
        start = free()
        s.adj_forward(SHORT, 10)
        assert 490 * MIB < start - free() < 520 * MIB
        s.adj_forward(LONG, 200)
        assert start - free() < 80 * MIB
        s.adj_forward(LONG, 2000)
        assert 490 * MIB < start - free() < 530 * MIB
        s.adj_forward(SHORT, 10)
        assert start - free() < 520 * MIB


@pytest.mark.gpu
def test_a_tape_takes_an_eighth_of_what_is_free(cuda):
    """With 3 GiB free the 0.5 GiB of states are not kept; with 6 GiB they are."""
    import torch

    p, v = ics.plummer(N, seed=1)
    torch.cuda.empty_cache()
    with NBodySystem(N, "f32", "sym", kick="physical", eps2=np.float32(1e-2), damping=1.0, dt=np.float32(1e-6)) as s:
        s.set_state(ics.f32(p), ics.f32(v))
        s.adj_forward(2, 1)
        fill = torch.empty((free() - 3 * GIB,), dtype=torch.uint8, device="cuda")
        start = free()
        s.adj_forward(SHORT, 100)
        assert start - free() < 60 * MIB
        del fill
        torch.cuda.empty_cache()
        fill = torch.empty((free() - 6 * GIB,), dtype=torch.uint8, device="cuda")
        start = free()
        s.adj_forward(SHORT, 100)
        assert start - free() > 430 * MIB
        del fill
        torch.cuda.empty_cache()
