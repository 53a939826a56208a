"""bench.py reports a kernel's captured DRAM traffic and pipe activity only for the kernel and
the size they were captured at."""
from __future__ import annotations

import bench


def test_captured_figures_are_not_scaled():
    at = {n: bench.ncu_capture("k_gsrb2", n) for n in (128, 224, 256, 512)}
    assert at[224] != at[256] and not at[128] and not at[512]
    for n in (224, 256):   # of 24 bytes per updated cell, what is left in the L2 of the array written does not move
        assert 0.75 < at[n]["dram_bytes"] / (12.0 * n ** 3) < 1.01 and 0 < at[n]["fp64_pipe_active"] < 1
    assert not bench.ncu_capture("k_gsrb", 256) and not bench.ncu_capture("k_gsrb_f4", 256)
