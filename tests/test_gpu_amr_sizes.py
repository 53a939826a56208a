"""The multilevel step at base grids whose rows are no power of two wide (blocks of other
than 256 threads in its kernels): one level against the single-level box, and two nested boxes against
the multilevel oracle.  Tolerances as in test_gpu_amr.py: positions 1e-14 against the box, 1e-12
against the oracle, the velocity change 1e-8 (both solves stop at rel_tol 1e-10)."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.amr import AmrHierarchy
from nyx_gb300.ics import zeldovich_ics
from nyx_gb300.pm import Box, Context
from oracle import oracle as O
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _step(ctx, vel, h, a0=0.05):
    dt = 0.4 * h * a0 / float(np.abs(vel).max())
    return a0, ctx.integrate_comoving_a(a0, dt), dt


@pytest.mark.parametrize("n0", [6, 8, 10, 12, 20, 24, 40, 48, 56, 80, 96, 112])
def test_one_level_equals_the_single_level_box(n0):
    ctx = Context()
    ic = zeldovich_ics(n0, 1.0, -2.0, 12, 0.05, rms_disp_cells=0.3)
    H = AmrHierarchy(ctx, n0, 1.0, [], len(ic.pos))
    B = Box(ctx, n0, 1.0, len(ic.pos))
    for x in (H, B):
        x.upload(ic.pos, ic.vel, ic.mass)
    step = _step(ctx, ic.vel, 1.0 / n0)
    # (the cycles differ: the box's new-time solve starts from its old field)
    H.step(*step)
    B.step(*step)
    (xa, va), (xb, vb) = H.download(), B.download()
    assert _rel(xa, xb) <= 1e-14
    assert _rel(va - ic.vel, vb - ic.vel) <= 1e-8


@pytest.mark.parametrize("n0", [20, 24, 28, 40, 48])
def test_nested_boxes_match_the_oracle(n0):
    ctx = Context()
    n = n0
    boxes = [[((n // 2,) * 3, (3 * n // 2 - 1,) * 3)], [((3 * n // 2,) * 3, (5 * n // 2 - 1,) * 3)]]
    ic = zeldovich_ics(n0, 1.0, -2.0, 31, 0.05, rms_disp_cells=0.4)
    H = AmrHierarchy(ctx, n0, 1.0, boxes, len(ic.pos))
    H.upload(ic.pos, ic.vel, ic.mass)
    p = O.Particles(ic.pos, ic.vel, ic.mass)
    A = O.AmrOracle(n0, 1.0, boxes, p)
    step = _step(ctx, ic.vel, 0.25 / n0)
    H.step(*step)
    A.step(*step)
    (x, v), (xo, vo) = H.download(), p.by_id()
    assert _rel(x, xo) <= 1e-12
    assert _rel(v - ic.vel, vo - ic.vel) <= 1e-8
