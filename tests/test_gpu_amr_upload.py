"""nyxpm_amr_upload's checks on the device: a value that is not finite is refused wherever
it stands, the first particle at fault names the reason, and a refused call leaves the
particles of the call before (exact)."""
from __future__ import annotations

import numpy as np
import pytest

from nyx_gb300.amr import AmrHierarchy
from nyx_gb300.pm import Box, Context, NyxPMError
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


@pytest.mark.parametrize("np_", [1, 33, 5003])
def test_refused_upload_names_the_first_fault_and_keeps_the_particles(np_):
    rng = np.random.default_rng(np_)
    pos, vel, mass = rng.random((np_, 3)), rng.normal(size=(np_, 3)), rng.random(np_)
    ctx = Context()
    H = AmrHierarchy(ctx, 8, 1.0, [], np_)
    H.upload(pos, vel, mass)
    last, mid = np_ - 1, np_ // 2
    faults = [((0, 0), None, "non-finite"), (None, (last, 2), "non-finite"), ((mid, 1), None, "non-finite")]
    for at_pos, at_vel, word in faults:
        for bad in (np.nan, np.inf, -np.inf):
            p, v = pos + 0.25, vel * 2
            for arr, at in ((p, at_pos), (v, at_vel)):
                if at:
                    arr[at] = bad
            for m in (mass, 1.0):
                with pytest.raises(NyxPMError, match=word):
                    H.upload(p, v, m)
    for m in (np.where(np.arange(np_) == last, -1.0, mass), np.where(np.arange(np_) == 0, np.nan, mass), -1.0, np.inf):
        with pytest.raises(NyxPMError, match="bad mass"):
            H.upload(pos + 0.25, vel * 2, m)
    if np_ > 1:     # a mass before a position: the mass is named
        p = pos.copy()
        p[last, 0] = np.nan
        with pytest.raises(NyxPMError, match="bad mass"):
            H.upload(p, vel, np.where(np.arange(np_) == 0, -1.0, mass))
    x, v = H.download()
    np.testing.assert_array_equal(x, pos)
    np.testing.assert_array_equal(v, vel)
    H.upload(pos, vel * 3, 2.0)
    np.testing.assert_array_equal(H.download()[1], vel * 3)


def test_masses_of_minus_zero_pass_and_others_out_of_range_do_not():
    """sum_masses: -0 is not negative; the largest number is finite (FP64 box and hierarchy)."""
    ctx = Context()
    rng = np.random.default_rng(3)
    pos, vel = rng.random((512, 3)), np.zeros((512, 3))
    box, H = Box(ctx, 8, 1.0, 512), AmrHierarchy(ctx, 8, 1.0, [], 512)
    for up in (box.upload, H.upload):
        for good in (-0.0, 0.0, 5e-324, 1.7e308):
            up(pos, vel, np.where(np.arange(512) == 300, good, 0.0))
        for bad in (-5e-324, -1.0, -np.inf, np.inf, np.nan, -np.nan):
            with pytest.raises(NyxPMError, match="bad mass"):
                up(pos, vel, np.where(np.arange(512) == 300, bad, 1.0))
