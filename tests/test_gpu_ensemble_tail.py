"""The two widths of the ensemble's coarse V-cycle kernel: boxes whose coarse levels start at
up to 32^3 (mg_fused_edge 8, 16, 24, 32) against one launch per pass (0), bit for bit
(tolerance: exact), with pre- and post-smoothing and without either.  With pre-smoothing the
boxes are powers of two: on a level whose rows hold no multiple of four compact cells the
launches restrict all eight children, the kernel the four red ones.
"""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ensemble import BoxSpec, Ensemble, box_ics
from nyx_gb300.pm import Context
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

SPECS = [BoxSpec(n, 0.5 if n % 3 else 1.0, n, -2.0) for n in (16, 20, 24, 28, 32, 48, 64)]
POWERS = [b for b in SPECS if b.n & (b.n - 1) == 0]


def _run(specs, edge, **kw):
    ctx = Context(mg_fused_edge=edge, **kw)
    ens = Ensemble(ctx, int(sum(1.05 * Ensemble.box_bytes(b.n, b.np) for b in specs)) + (32 << 20))
    slots = []
    for b in specs:
        ic = box_ics(b)
        slots.append(ens.add(b.n, b.L, b.np))
        ens.upload(slots[-1], ic.pos, ic.vel, ic.mass)
    for a0, a1, dt in ctx.step_schedule(0.02, 0.04, 2):
        ens.step({s: a0 for s in slots}, {s: a1 for s in slots}, {s: dt for s in slots})
    out = [(*ens.download(s), ens.get_phi(s)) for s in slots]
    ens.close()
    ctx.close()
    return out


@pytest.mark.parametrize("specs, kw", [(POWERS, {}), (POWERS, {"nu1": 4, "nu2": 0}), (SPECS, {"nu1": 0, "nu2": 4})])
def test_coarse_levels_in_one_kernel_equal_launches(specs, kw):
    expect = _run(specs, 0, **kw)
    for edge in (8, 16, 24, 32):
        for box, got in zip(expect, _run(specs, edge, **kw)):
            for x, y in zip(box, got):
                np.testing.assert_array_equal(x, y)
