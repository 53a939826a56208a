"""Boxes whose solve is one cluster launch, and boxes whose coarse levels are one
(nyx_gb300/csrc/pm_cluster.cuh), against one launch per pass (mg_fused_edge = 0), bit for bit
(tolerance: exact): the cycle limit, other sweep counts, an empty right-hand side, a solve from
the last step's phi.  That the cluster is what runs shows in the number of launches.

A whole box is taken up to 32^3 in FP64 and 48^3 in FP32, below a finest level 16^3 and 32^3;
a slab has one to three planes (48 on 16 CTAs), uneven at 20, 24 and 40; the FP64 levels of
one CTA start at 8^3, so that 10^3 and 14^3 and what coarsens to them go by launches.
"""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ics import zeldovich_ics
from nyx_gb300.pm import Box, Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

WHOLE = [("fp64", n) for n in (12, 16, 24, 32)] + [("mixed", n) for n in (20, 24, 28, 32, 40, 48)]
BELOW = [("fp64", n) for n in (48, 64, 96)] + [("mixed", n) for n in (56, 64, 80, 96)]


def _run(precision, n, steps, lattice, **kw):
    ctx = Context(**kw)
    ic = zeldovich_ics(n, 1.0, -2.0, 5, 0.05, rms_disp_cells=0.4)
    box = Box(ctx, n, 1.0, len(ic.pos), precision=precision)
    box.upload(ic.lattice if lattice else ic.pos, ic.vel, ic.mass)
    before, infos, a = ctx.launch_count(), [], 0.05
    for _ in range(steps):
        try:
            infos.append(box.step(a, a + 0.01, ctx.step_schedule(a, a + 0.01, 1)[0][2]))
        except NyxPMError:
            infos.append("above tolerance")
        a += 0.01
    launches = ctx.launch_count() - before
    out = (*box.download(), box.get_phi(), box.grav_vector())
    box.close()
    ctx.close()
    return out, infos, launches


def _same(precision, n, steps=2, lattice=False, **kw):
    got, infos, few = _run(precision, n, steps, lattice, **kw)
    expect, expected, many = _run(precision, n, steps, lattice, mg_fused_edge=0, **kw)
    assert infos == expected
    for x, y in zip(got, expect):
        np.testing.assert_array_equal(x, y)
    return infos, few, many


@pytest.mark.parametrize("precision, n", WHOLE)
def test_whole_box(precision, n):
    infos, few, many = _same(precision, n)
    assert 4 * few < many and "above tolerance" not in infos
    infos, few, many = _same(precision, n, max_vcycles=1)   # stops above tolerance
    assert few < many and infos == 2 * ["above tolerance"]
    for nu1, nu2 in ((1, 3), (3, 1)):
        infos, few, many = _same(precision, n, nu1=nu1, nu2=nu2)
        assert 4 * few < many and "above tolerance" not in infos
    infos, few, many = _same(precision, n, steps=1, lattice=True)
    assert "above tolerance" not in infos


@pytest.mark.parametrize("precision, n", BELOW)
def test_coarse_levels(precision, n):
    infos, few, many = _same(precision, n)
    assert few < many and "above tolerance" not in infos
    infos, few, many = _same(precision, n, nu1=1, nu2=3)
    assert few < many and "above tolerance" not in infos
