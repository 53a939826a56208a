"""The read-back that the host polls for (post_open / post_words / post_wait): solves
that follow one another on one stream, alternating between boxes and after a solve that
stopped at its cycle limit, each report the norms and cycles that the same solve reports
alone in a fresh context (exact)."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ics import zeldovich_ics
from nyx_gb300.pm import Box, Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _box(ctx, n, precision, seed):
    ic = zeldovich_ics(n, 1.0, -2.0, seed, 0.05, rms_disp_cells=0.4)
    box = Box(ctx, n, 1.0, len(ic.pos), precision=precision)
    box.upload(ic.pos, ic.vel, ic.mass)
    return box


def _step(ctx, box, k):
    a = 0.05 + 0.01 * k
    try:
        info = box.step(a, a + 0.01, ctx.step_schedule(a, a + 0.01, 1)[0][2])
    except NyxPMError:
        info = "limit"
    return info, box.est_time_step(0.5, a + 0.01)


@pytest.mark.parametrize("kw", [{}, {"max_vcycles": 3}, {"mg_fused_edge": 0}], ids=["", "limit", "launches"])
def test_boxes_in_turn_report_what_each_reports_alone(kw):
    forms = [(48, "fp64", 3), (16, "fp64", 4), (80, "mixed", 5), (32, "mixed", 6)]
    ctx = Context(**kw)
    boxes = [_box(ctx, *f) for f in forms]
    turns = [[_step(ctx, b, k) for b in boxes] for k in range(3)]
    for i, f in enumerate(forms):
        alone = Context(**kw)
        box = _box(alone, *f)
        assert [t[i] for t in turns] == [_step(alone, box, k) for k in range(3)]
        for x, y in zip(box.download(), boxes[i].download()):
            np.testing.assert_array_equal(x, y)
