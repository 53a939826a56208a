"""The allocation-free deposit at the sizes where its two paths change, against the same sums
in numpy, bit for bit (tolerance: exact): grids that are no multiple of the 8 x 8 x 4 tile and
smaller than it, the last and the first grid and particle count on either side of the cluster
sort (131,072 cells or particles), keys of 32, 33, 512, 513 and thousands of particles, and one
non-finite position on each path.

The box's side is n, so that a position in cells is x + 1/2 rounded once.  A key's particles
are added in their order; a key of more than 32 by 32 lanes (lane l: particles l, l + 32, ...)
and an xor butterfly; a cell adds its eight keys' corners z slowest, x fastest.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from nyx_gb300 import _lib
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]

MASS = 1.5


def _positions(n, np_, clumps, seed):
    rng = np.random.default_rng(seed)
    pos = rng.random((np_, 3)) * n
    at = 0
    for size in clumps:   # all of a clump in one key
        key = rng.integers(0, n, 3)
        pos[at:at + size] = np.mod(key + 0.99 * rng.random((size, 3)) - 0.5, n)
        at += size
    return np.minimum(pos[rng.permutation(np_)], np.nextafter(n, 0))


def _reference(n, pos):
    l = pos + 0.5
    cell = np.floor(l)
    frac = l - cell
    cell = np.mod(cell.astype(np.int64), n)
    key = cell[:, 0] + n * (cell[:, 1] + n * cell[:, 2])
    order = np.argsort(key, kind="stable")
    s = np.stack([1.0 - frac, frac])[:, order]   # [complement or fraction][particle][axis]
    w = np.stack([(s[c & 1, :, 0] * s[c >> 1 & 1, :, 1]) * s[c >> 2, :, 2] for c in range(8)], axis=1)
    count = np.bincount(key, minlength=n ** 3)
    start = np.concatenate([[0], np.cumsum(count)])
    part = np.zeros((n ** 3, 8))
    for t in range(32):
        K = np.nonzero((count > t) & (count <= 32))[0]
        part[K] = part[K] + w[start[K] + t]
    for K in np.nonzero(count > 32)[0]:
        lanes = np.zeros((32, 8))
        for q in range(0, count[K], 32):
            m = min(32, count[K] - q)
            lanes[:m] = lanes[:m] + w[start[K] + q:start[K] + q + m]
        for off in (16, 8, 4, 2, 1):
            lanes = lanes + lanes[np.arange(32) ^ off]
        part[K] = lanes[0]
    part = part.reshape(n, n, n, 8)
    rho = np.zeros((n, n, n))
    for d in range(8):
        di, dj, dk = d & 1, d >> 1 & 1, d >> 2
        rho = rho + np.roll(part[..., (1 - di) + 2 * (1 - dj) + 4 * (1 - dk)], (-dk, -dj, -di), (0, 1, 2))
    return (rho * MASS).reshape(-1)


@pytest.mark.parametrize("n, np_, clumps", [
    (4, 1, []), (4, 64, [33]), (10, 2000, [32, 33, 513]), (14, 131072, []), (28, 50001, [512, 513, 4097]),
    (50, 131072, [33, 9000]), (51, 131072, [33, 512, 9000]), (51, 1000, [33, 64]), (32, 131073, [32, 513, 5000]),
    (64, 262144, [33, 512, 513, 20000])])
def test_deposit_equals_the_ordered_sums(n, np_, clumps):
    import torch
    lib, err = _lib.load(), C.create_string_buffer(256)
    pos = _positions(n, np_, clumps, 7 * n + np_)
    x, y, z = (torch.tensor(np.ascontiguousarray(pos[:, d]), device="cuda") for d in range(3))
    rho = torch.full((n ** 3,), float("nan"), dtype=torch.float64, device="cuda")

    def call():
        return lib.nyxpm_deposit_noalloc(x.data_ptr(), y.data_ptr(), z.data_ptr(), np_, MASS, n, float(n),
                                         rho.data_ptr(), torch.cuda.current_stream().cuda_stream, err, len(err))

    expect = _reference(n, pos)
    for _ in range(2):   # again over the scratch the call before left
        rho.fill_(float("nan"))
        assert call() == 0, err.value
        np.testing.assert_array_equal(rho.cpu().numpy(), expect)
    y[np_ - 1] = float("nan")
    assert call() == 1 and b"non-finite" in err.value
