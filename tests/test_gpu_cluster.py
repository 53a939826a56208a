"""Small levels cycled by one thread-block cluster (nyx_gb300/csrc/pm_cluster.cuh) against
one launch per pass (mg_fused_edge = 0), bit for bit (tolerance: exact), at every edge
the cluster takes as the finest level and at edges that reach it after one or two
launches: slabs of one to four planes, uneven slabs (20, 24, 28, 40, 56 planes on 16
CTAs), levels of odd and even halves, bottoms of 3, 4, 5 and 7 cells.
"""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ics import zeldovich_ics
from nyx_gb300.pm import Box, Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _solve(n, precision, steps=2, pos=None, **kw):
    ctx = Context(**kw)
    ic = zeldovich_ics(n, 1.0, -2.0, 7, 0.05, rms_disp_cells=0.4)
    box = Box(ctx, n, 1.0, len(ic.pos), precision=precision)
    box.upload(ic.lattice if pos == "lattice" else ic.pos, ic.vel, ic.mass)
    infos, failed = [], 0
    a = 0.05
    for _ in range(steps):
        try:
            infos.append(box.step(a, a + 0.01, ctx.step_schedule(a, a + 0.01, 1)[0][2]))
        except NyxPMError:
            failed += 1
        a += 0.01
    out = (*box.download(), box.get_phi())
    box.close()
    return out, infos, failed


def _same(n, precision, **kw):
    (a, ia, fa), (b, ib, fb) = (_solve(n, precision, **{**kw, **e}) for e in ({}, {"mg_fused_edge": 0}))
    assert ia == ib and fa == fb
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    return fa


@pytest.mark.parametrize("n", [10, 12, 16, 20, 24, 32, 40, 48, 64])
def test_fp64_cluster_equals_launches(n):
    assert _same(n, "fp64") == 0


@pytest.mark.parametrize("n", [20, 24, 28, 32, 40, 48, 56, 64, 80, 96, 112])
def test_mixed_cluster_equals_launches(n):
    assert _same(n, "mixed") == 0


@pytest.mark.parametrize("precision, n", [("fp64", 32), ("mixed", 64)])
def test_cycle_limit_other_sweeps_and_an_empty_right_hand_side(precision, n):
    assert _same(n, precision, max_vcycles=2) == 2      # stops above tolerance
    assert _same(n, precision, nu1=1, nu2=3) == 0
    assert _same(n, precision, pos="lattice", steps=1) == 0
