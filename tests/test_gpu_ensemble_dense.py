"""Ensemble boxes with many particles per cell: particles go in and out in a number of pieces
that does not grow with np / n^3, through the particle buffer that is not current, and a
download leaves the box as it was (tolerances: bits exact; times, a factor of 5)."""
from __future__ import annotations

import time

import numpy as np
import pytest

from nyx_gb300.ensemble import Ensemble
from nyx_gb300.pm import Context
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _particles(np_, seed):
    rng = np.random.default_rng(seed)
    return rng.random((np_, 3)), rng.normal(0, 300.0, (np_, 3))


def _times(n, np_):
    ctx = Context()
    ens = Ensemble(ctx, Ensemble.box_bytes(n, np_) + (8 << 20))
    slot = ens.add(n, 1.0, np_)
    pos, vel = _particles(np_, n)
    up, down = [], []
    for _ in range(5):
        t = time.perf_counter()
        ens.upload(slot, pos, vel, 1.0e9)
        up.append(time.perf_counter() - t)
        t = time.perf_counter()
        ens.download(slot)
        down.append(time.perf_counter() - t)
    ens.close()
    ctx.close()
    return min(up), min(down)


def test_as_fast_on_a_coarse_grid_as_on_a_fine_one():
    coarse, fine = _times(16, 1000000), _times(96, 1000000)
    assert coarse[0] < 5 * fine[0] and coarse[1] < 5 * fine[1], (coarse, fine)


@pytest.mark.parametrize("np_", [4096, 4097, 9001, 60000])
def test_a_download_between_steps_changes_nothing(np_):
    pos, vel = _particles(np_, np_)
    out = []
    for look in (False, True):
        ctx = Context()
        ens = Ensemble(ctx, Ensemble.box_bytes(16, np_) + (8 << 20))
        slot = ens.add(16, 1.0, np_)
        ens.upload(slot, pos, vel, 1.0e9)
        for a0, a1, dt in ctx.step_schedule(0.5, 0.503, 3):
            if look:
                first, again = ens.download(slot), ens.download(slot)
                for x, y in zip(first, again):
                    np.testing.assert_array_equal(x, y)
            ens.step({slot: a0}, {slot: a1}, {slot: dt})
        out.append((*ens.download(slot), ens.get_phi(slot), ens.grav_vector(slot)))
        ens.close()
        ctx.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
