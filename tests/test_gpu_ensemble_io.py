"""Ensemble particles in and out (nyxpm_ensemble_upload / _download, converted on the
device in pieces of n^3 / 6 particles) against the same conversion in numpy, bit for bit
(tolerance: exact): fewer particles than a piece, a piece and one more, more particles
than cells; positions on, just below and just above cell edges, outside the box, and the
offsets that round up to the next cell's origin."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ensemble import Ensemble
from nyx_gb300.pm import Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _expect(pos, n, L):
    l = pos * (n / L)
    fl = np.floor(l)
    o = (l - fl).astype(np.float32)
    up = o >= 1.0
    o[up] = 0.0
    return (np.mod(fl + up, n) + o.astype(np.float64)) * (L / n)


@pytest.mark.parametrize("n, np_, L", [(16, 1, 1.0), (16, 682, 1.0), (16, 683, 7.5), (16, 5001, 1.0),
                                       (24, 13824, 0.3), (40, 32001, 1.0)])
def test_round_trip_equals_the_conversion(n, np_, L):
    rng = np.random.default_rng(n + np_)
    pos = rng.uniform(-0.5 * L, 1.5 * L, (np_, 3))
    edge = (rng.integers(0, n + 1, (np_, 3)) * (L / n)) * (1.0 + rng.integers(-2, 3, (np_, 3)) * 2.0 ** -52)
    pos = np.where(rng.random((np_, 3)) < 0.3, edge, pos)
    vel = rng.normal(0, 300.0, (np_, 3))
    ens = Ensemble(Context(), Ensemble.box_bytes(n, np_) + (8 << 20))
    slot = ens.add(n, L, np_)
    for _ in range(2):   # again into a slot that holds particles
        ens.upload(slot, pos, vel, 1.0e9)
        p, v = ens.download(slot)
        np.testing.assert_array_equal(p, _expect(pos, n, L))
        np.testing.assert_array_equal(v, vel.astype(np.float32).astype(np.float64))
        pos, vel = pos[::-1].copy(), vel[::-1].copy()
    bad = pos.copy()
    bad[np_ // 2, 1] = np.inf
    with pytest.raises(NyxPMError):
        ens.upload(slot, bad, vel, 1.0e9)
    with pytest.raises(NyxPMError):   # refused particles leave the slot without any
        ens.download(slot)
    ens.close()
