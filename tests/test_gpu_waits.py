"""An application that asks the device for blocking waits (cudaSetDeviceFlags) has its thread's
CPU back while a solve or the allocation-free deposit waits: in a child process, the thread's
CPU time against the wall time.  A wait here is a millisecond and more of device time;
tolerance: half the wall time (a poll takes all of it).  Yielding gives the CPU away to others
only, so that it is run and not timed.
"""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from tests.conftest import REPO, gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

CHILD = r"""
import ctypes as C, sys, time
import numpy as np
from nyx_gb300 import _lib
lib = _lib.load()
assert C.CDLL("libcudart.so.13").cudaSetDeviceFlags(int(sys.argv[1])) == 0
import torch
from nyx_gb300.pm import Box, Context

share = {}

def timed(name, call, repeats):
    call()
    torch.cuda.synchronize()
    t, w = time.thread_time(), time.perf_counter()
    for _ in range(repeats):
        call()
    share[name] = (time.thread_time() - t) / (time.perf_counter() - w)

pos = np.random.default_rng(2).random((4096, 3))
ctx = Context(device=0)
for form in ("fp64", "mixed"):
    box = Box(ctx, 256, 1.0, len(pos), precision=form)
    box.upload(pos, np.zeros_like(pos), 1.0e12)
    box.deposit(read_back=False)
    info = box.solve_phi(0.5, zero_guess=True)
    assert info["vcycles"] > 3, info
    timed(form, lambda: box.solve_phi(0.5, zero_guess=True), 8)
    box.close()

err = C.create_string_buffer(256)
x = torch.rand(1000, device="cuda", dtype=torch.float64)
rho = torch.empty(16 ** 3, device="cuda", dtype=torch.float64)
a = torch.randn(4096, 4096, device="cuda")
b = torch.empty_like(a)

def deposit():   # behind some milliseconds of other work on the stream
    for _ in range(20):
        torch.mm(a, a, out=b)
    st = lib.nyxpm_deposit_noalloc(x.data_ptr(), x.data_ptr(), x.data_ptr(), 1000, 1.0, 16, 1.0, rho.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream, err, len(err))
    assert st == 0, err.value

timed("noalloc", deposit, 8)
assert abs(float(rho.sum()) / (1000 * 16 ** 3) - 1) < 1e-12
print(" ".join(f"{k} {v:.3f}" for k, v in share.items()))
"""


def _child(flags):
    env = {**os.environ, "PYTHONPATH": os.pathsep.join([REPO, os.environ.get("PYTHONPATH", "")])}
    r = subprocess.run([sys.executable, "-c", CHILD, str(flags)], cwd=REPO, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    words = r.stdout.split()
    return dict(zip(words[::2], map(float, words[1::2])))


def test_blocking_waits_give_the_cpu_away():
    share = _child(4)
    assert set(share) == {"fp64", "mixed", "noalloc"} and max(share.values()) < 0.5, share


@pytest.mark.parametrize("flags", [1, 2])   # spin, yield
def test_other_waits(flags):
    assert set(_child(flags)) == {"fp64", "mixed", "noalloc"}
