"""FP64 solves from a zero guess take the right-hand side for their residual and do not read
phi (mg_solve's from_zero): after an earlier solve has left a field behind, a solve from a zero
guess gives what a fresh box gives, bit for bit, in the cluster, by launches, without
pre- or post-smoothing (the general path), at a cycle limit and for a uniform density (no
right-hand side: phi = 0)."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.ics import zeldovich_ics
from nyx_gb300.pm import Box, Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _solve(box):
    box.deposit(read_back=False)
    try:
        info = box.solve_phi(0.05, zero_guess=True)
    except NyxPMError:
        info = "limit"
    return info, box.get_phi(), box.grav_vector()


@pytest.mark.parametrize("kw", [{}, {"mg_fused_edge": 0}, {"nu1": 0}, {"nu2": 0}, {"nu1": 1, "nu2": 1},
                                {"max_vcycles": 1}], ids=str)
@pytest.mark.parametrize("n", [4, 12, 32, 40, 96])
def test_zero_guess_does_not_see_the_field_before(n, kw):
    ic = zeldovich_ics(n, 1.0, -2.0, 3, 0.05, rms_disp_cells=0.6)
    lattice = np.stack(np.meshgrid(*[(np.arange(n) + 0.5) / n] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(n)
    used = Box(Context(**kw), n, 1.0, n ** 3)
    for pos in (rng.random((n ** 3, 3)), ic.pos, lattice):
        fresh = Box(Context(**kw), n, 1.0, n ** 3)
        for b in (used, fresh):
            b.upload(pos, ic.vel, ic.mass)
        (ia, pa, ga), (ib, pb, gb) = _solve(used), _solve(fresh)
        assert ia == ib
        np.testing.assert_array_equal(pa, pb)
        np.testing.assert_array_equal(ga, gb)
        if pos is lattice and n & (n - 1) == 0:   # corner weights of 1/2 add up to 1 exactly
            assert not pa.any() and not ga.any()
