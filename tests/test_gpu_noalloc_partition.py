"""The allocation-free deposit where a cluster of 16 CTAs cannot be placed (an SM partition,
say): the call sorts by launches and gives nyxpm_deposit's density, bit for bit (tolerance:
exact).  The device that cannot place it is a host-side stand-in for two runtime calls,
preloaded into a child process: the occupancy query answers 0 clusters (or 1: only the
launch refuses then), and a launch that asks for a cluster of 16 returns
cudaErrorInvalidClusterSize.  Every other call goes to the runtime.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

import pytest

from tests.conftest import REPO, gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

STAND_IN = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdlib.h>

cudaError_t cudaOccupancyMaxActiveClusters(int *clusters, const void *func, const cudaLaunchConfig_t *cfg)
{
    (void)func, (void)cfg;
    *clusters = atoi(getenv("PLACED_CLUSTERS"));
    return cudaSuccess;
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *func, void **args)
{
    static cudaError_t (*launch)(const cudaLaunchConfig_t *, const void *, void **);
    for (unsigned i = 0; i < cfg->numAttrs; ++i)
        if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension && cfg->attrs[i].val.clusterDim.x >= 16)
            return cudaErrorInvalidClusterSize;
    if (!launch) *(void **)&launch = dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    return launch(cfg, func, args);
}
"""

CHILD = r"""
import ctypes as C
import numpy as np
import torch
from nyx_gb300 import _lib
from nyx_gb300.pm import Box, Context

lib, ctx, err = _lib.load(), Context(device=0), C.create_string_buffer(256)
rng = np.random.default_rng(3)
for n, np_ in [(1, 1), (10, 700), (32, 32768), (48, 131072)]:
    pos = np.concatenate([rng.random((np_ - np_ // 4, 3)), 0.4 + 0.01 * rng.random((np_ // 4, 3))])
    x, y, z = (torch.tensor(np.ascontiguousarray(pos[:, d]), device="cuda") for d in range(3))
    rho = torch.full((n ** 3,), float("nan"), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def call():
        return lib.nyxpm_deposit_noalloc(x.data_ptr(), y.data_ptr(), z.data_ptr(), np_, 2.0e9, n, 1.0,
                                         rho.data_ptr(), stream, err, len(err))

    for _ in range(2):
        assert call() == 0, err.value
    if n > 1:
        box = Box(ctx, n, 1.0, np_)
        box.upload(pos, np.zeros_like(pos), 2.0e9)
        assert np.array_equal(rho.cpu().numpy(), box.deposit())
        box.close()
    assert abs(float(rho.sum()) - 2.0e9 * np_ * n ** 3) < 1e-9 * 2.0e9 * np_ * n ** 3
    x[np_ // 2] = float("inf")
    assert call() == 1 and b"non-finite" in err.value
print("ok")
"""


@pytest.mark.parametrize("placed", ["0", "1"])
def test_without_a_place_for_the_cluster(tmp_path, placed):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    roots = ("include", "targets/sbsa-linux/include", "targets/x86_64-linux/include")
    include = [f"-I{os.path.join(cuda, d)}" for d in roots]
    src, so = tmp_path / "stand_in.c", tmp_path / "stand_in.so"
    src.write_text(STAND_IN)
    subprocess.run(["gcc", "-shared", "-fPIC", *include, "-o", str(so), str(src), "-ldl"], check=True)
    env = {**os.environ, "LD_PRELOAD": str(so), "PLACED_CLUSTERS": placed,
           "PYTHONPATH": os.pathsep.join([REPO, os.environ.get("PYTHONPATH", "")])}
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=REPO, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-4000:]
