"""The cloud-in-cell weights and products on the integer pipe (pm_cic.cuh) in the FP64
deposit and kicks against the oracle, bit for bit (tolerance: exact): positions on cell
faces and centres, a few last places off them, next to 0 and to the box's edge, and
random; keys of one to many particles; accelerations of every sign, zero, subnormal-sized
and of a single bit."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.pm import Box, Context
from oracle import oracle as O
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _positions(n, L, rng):
    h = L / n
    faces = (rng.integers(0, n, (300, 3)) + rng.choice([0.0, 0.5], (300, 3))) * h
    off = faces + rng.integers(-3, 4, faces.shape) * np.spacing(np.maximum(faces, h))
    tiny = np.concatenate([rng.random((40, 3)) * 10.0 ** rng.uniform(-300, -1, (40, 1)),
                           L - L * 10.0 ** rng.uniform(-16, -1, (40, 3))])
    clump = L * (0.37 + 0.2 * h * rng.random((150, 3)))
    sparse = np.ldexp(rng.integers(0, 64, (200, 3)), -6) * L
    pos = np.concatenate([faces, off, tiny, clump, sparse, rng.random((4 * n * n, 3)) * L])
    return np.where((pos < 0) | (pos >= L), 0.0, pos)


@pytest.mark.parametrize("masses", [False, True])
@pytest.mark.parametrize("n, L", [(8, 1.0), (20, 0.7), (64, 28.49002849)])
def test_deposit_and_kicks_equal_the_oracle(n, L, masses):
    rng = np.random.default_rng(n)
    pos = _positions(n, L, rng)
    vel = rng.normal(size=pos.shape) * L * 10.0 ** rng.uniform(-12, 1, pos.shape)
    mass = rng.random(len(pos)) + 0.5 if masses else 1.25
    box = Box(Context(), n, L, len(pos))
    box.upload(pos, vel, mass)
    p = O.Particles(pos, vel, mass)
    np.testing.assert_array_equal(box.deposit().ravel(), O.deposit(n, L, p, O.sort(n, L, p)).ravel())
    g = rng.normal(size=3 * n ** 3) * 10.0 ** rng.uniform(-20, 3, 3 * n ** 3)
    kind = rng.integers(0, 8, g.size)
    g[kind == 0] = 0.0
    g[kind == 1] = np.ldexp(np.sign(g[kind == 1]), rng.integers(-60, 3, (kind == 1).sum()))
    g[: n * n] *= 1e-300
    box.set_grav_vector(g)
    dt, a, a_half, a_new = 3e-3, 0.3, 0.31, 0.33
    box.kick_drift(dt, a, a_half)
    O.move(n, L, p, g, dt, a, a_half, 1)
    for x, y in zip(box.download(), p.by_id()):
        np.testing.assert_array_equal(x, y)
    box.kick(dt, a_new, a_half)
    O.move(n, L, p, g, dt, a_half, a_new, 0)
    for x, y in zip(box.download(), p.by_id()):
        np.testing.assert_array_equal(x, y)
