"""GPU parity of the shared-memory QR kernels (qr_smem.cuh: geqrf and gels beyond the register kernels),
bit for bit against the CPU oracle at the edges of a lane's columns, of a warp's 64 columns, of the
256-column and the shared-memory limits, with zero, infinite and NaN members and padding."""
from __future__ import annotations

import numpy as np
import pytest

from test_gels_gpu import check as check_gels
from test_geqrf_gpu import check as check_geqrf

pytestmark = pytest.mark.gpu


def _members(rng, shape, m):
    a = rng.standard_normal(shape).astype(np.float32)
    n = shape[1]
    a[1, :, :m] = 0.0
    a[2, n // 2, :m] = 0.0
    a[3, n // 3, m // 2] = np.inf
    a[4, n // 2, m // 3] = np.nan
    a[5, :, 1:m] = 0.0  # nothing below the first row
    return a


@pytest.mark.parametrize("mn", [(33, 1), (1, 33), (33, 2), (2, 33), (33, 32), (32, 33), (64, 48), (47, 64), (65, 65), (64, 66), (40, 128),
                                (129, 40), (30, 129), (35, 193), (20, 256), (20, 257), (222, 222), (256, 200)])
def test_geqrf_smem_edges(handle, mn):
    m, n = mn
    for lda in (m, m + 5):
        a = _members(np.random.default_rng(m * 300 + n), (7, n, lda), m)
        with np.errstate(all="ignore"):
            check_geqrf(handle, a, m, n, lda, f"{m}x{n} lda {lda}")


@pytest.mark.parametrize("batch", [7, 200])
def test_gels_one_column(handle, batch):
    """One reflector: in global memory for a small batch, in shared memory for one that fills the GPU."""
    rng = np.random.default_rng(batch)
    a = _members(rng, (batch, 1, 33), 33)
    c = rng.standard_normal((batch, 20, 33)).astype(np.float32)
    with np.errstate(all="ignore"):
        check_gels(handle, "N", a, c, 33, 1, 20, 33, 33, f"33x1 batch {batch}")


@pytest.mark.parametrize("shape", [("N", 33, 32, 1), ("N", 64, 48, 15), ("N", 64, 48, 17), ("T", 48, 64, 1),
                                   ("N", 65, 65, 64), ("N", 40, 1, 255), ("N", 40, 1, 256), ("T", 20, 100, 40),
                                   ("N", 150, 100, 130), ("N", 220, 200, 3), ("N", 260, 200, 3)])
def test_gels_smem_edges(handle, shape):
    t, m, n, nrhs = shape
    rng = np.random.default_rng(m * 131 + n * 7 + nrhs)
    for pad in (0, 3):
        lda, ldc = m + pad, max(m, n) + pad
        a = _members(rng, (7, n, lda), m)
        c = rng.standard_normal((7, nrhs, ldc)).astype(np.float32)
        c[6, nrhs // 2, 0] = np.nan
        with np.errstate(all="ignore"):
            check_gels(handle, t, a, c, m, n, nrhs, lda, ldc, f"{t} {m}x{n}x{nrhs} pad {pad}")
