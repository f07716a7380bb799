"""GPU parity of the blocked kernels for 32 < n <= 256: the shared-memory LU (getrf_mid.cu, n <= 128)
and the block inverse (getri_block_kernel). Bit for bit against the CPU oracle at the edges of their
blocks of 16 columns and tiles of 32 rows."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import to_dev, to_host
from test_lu_gpu import assert_bitwise, gpu_getrf, gpu_getri

pytestmark = pytest.mark.gpu

EDGES = [33, 47, 48, 49, 63, 64, 65, 79, 81, 96, 97, 100, 112, 113, 127, 128]


def _check_getrf(handle, a, n, lda, pivot=True):
    lu, piv, info = gpu_getrf(handle, a, n, lda, pivot=pivot)
    olu = a.copy()
    opiv, oinfo, _ = O.port_getrf(olu, n, lda, pivot=pivot)
    assert_bitwise(lu, olu, f"LU n={n} lda={lda}")
    if pivot:
        np.testing.assert_array_equal(piv, opiv)
    np.testing.assert_array_equal(info, oinfo)
    return info


@pytest.mark.parametrize("n", EDGES)
def test_getrf_block_edges(handle, n):
    """Random, tied, scaled (the quotients' range limits) and non-finite matrices; padded rows."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((12, n, n)).astype(np.float32)
    a[1] = np.round(a[1])                                    # exact ties and signed zeros
    a[2] = np.sign(a[2])                                     # ties in every column
    a[3] *= np.float32(2.0 ** -70)                           # pivots below the shared-reciprocal range
    a[4] *= np.float32(2.0 ** 70)                            # and above
    a[5] *= np.exp2(rng.integers(-64, 64, (n, n))).astype(np.float32)
    a[6] *= np.exp2(rng.integers(-140, -100, (n, n))).astype(np.float32)  # subnormals
    a[7, n // 3, n // 2] = np.nan
    a[8, n // 2, n // 3] = np.inf
    a[9] = np.where(rng.random((n, n)) < 0.8, 0.0, a[9])     # sparse: zero multipliers
    a[10] = np.eye(n, dtype=np.float32)[::-1] * -1.0
    a[11, 3] = np.nan                                        # a column without a candidate
    with np.errstate(all="ignore"):
        _check_getrf(handle, a, n, n)
        b = rng.standard_normal((3, n, n + 4)).astype(np.float32)
        b[:, :, n:] = 77.0
        _check_getrf(handle, b, n, n + 4)
        c = rng.standard_normal((3, n, n + 1)).astype(np.float32)
        _check_getrf(handle, c, n, n + 1)


@pytest.mark.parametrize("n", [40, 64, 90, 128])
def test_getrf_stops(handle, n):
    """Zero columns on both sides of block boundaries: info, positions kept and pivots zeroed past the stop."""
    cols = sorted({0, 1, 15, 16, 17, 31, 32, n // 2, n - 2, n - 1})
    rng = np.random.default_rng(n + 7)
    a = rng.standard_normal((len(cols), n, n)).astype(np.float32)
    for q, c in enumerate(cols):
        a[q, c] = 0.0
    assert list(_check_getrf(handle, a, n, n)) == [c + 1 for c in cols]
    d = rng.standard_normal((2, n, n)).astype(np.float32) + 2 * n * np.eye(n, dtype=np.float32)
    d[1, n // 2] = 0.0
    _check_getrf(handle, d, n, n, pivot=False)


@pytest.mark.parametrize("n", EDGES + [129, 144, 161, 192, 193, 255, 256])
def test_getri_block_edges(handle, n):
    """Inverses with interchanges, padded and odd strides, a zero on the diagonal of each kind of panel."""
    rng = np.random.default_rng(3 * n)
    for lda, ldc, batch in ((n, n, 6), (n + 4, n + 1, 2), (n + 1, n + 4, 2)):
        lu = rng.standard_normal((batch, n, lda)).astype(np.float32)
        lu[:, np.arange(n), np.arange(n)] += np.where(rng.random(n) < 0.5, -8, 8)
        piv = np.stack([np.arange(1, n + 1) + rng.integers(0, n - np.arange(n)) for _ in range(batch)]).astype(np.int32)
        if batch == 6:
            lu[1, 0, 0] = 0.0
            lu[2, n - 1, n - 1] = 0.0
            lu[3, 16, 16] = 0.0
            lu[4, 15, 15] = 0.0
            lu[5, 2, 5] = np.inf
        c, info = gpu_getri(handle, lu, n, lda, piv, ldc)
        oc = np.full((batch, n, ldc), -7.0, np.float32)
        with np.errstate(all="ignore"):
            oinfo = O.port_getri(lu, n, lda, piv, oc, ldc)
        np.testing.assert_array_equal(info, oinfo)
        assert_bitwise(c, oc, f"C n={n} lda={lda}")
    c, info = gpu_getri(handle, lu, n, lda, None, ldc)
    oc = np.full((batch, n, ldc), -7.0, np.float32)
    oinfo = O.port_getri(lu, n, lda, None, oc, ldc)
    assert_bitwise(c, oc, f"C n={n} without pivots")


@pytest.mark.parametrize("n", [33, 40, 63, 64, 65, 72, 96, 97, 104, 127, 128])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_getrs_staged_edges(handle, n, trans):
    """The staged solve (getrs_staged.cu): block and tile edges, column counts on both sides of its warp and CTA
    limits, odd strides, invalid pivots, zeros, infinities and NaN in the right-hand sides."""
    rng = np.random.default_rng(n)
    for nrhs, batch, pad in ((1, 5, 0), (2, 3, 1), (3, 37, 0), (8, 9, 4), (17, 2, 0), (33, 2, 3), (130, 1, 0)):
        ld = n + pad
        lu = rng.standard_normal((batch, n, ld)).astype(np.float32)
        piv, _, _ = O.port_getrf(lu, n, ld)
        piv[0, 0] = 0
        piv[0, n - 1] = n + 7
        b = rng.standard_normal((batch, nrhs, ld)).astype(np.float32)
        b[0, 0, : n // 2] = 0.0
        if nrhs > 2:
            b[batch - 1, 1, n - 1] = np.inf
            b[batch - 1, 2, 0] = np.nan
        want = b.copy()
        with np.errstate(all="ignore"):
            O.port_getrs(trans, lu, n, ld, piv, want, nrhs, ld)
        B = to_dev(b, "cuda")
        handle.getrs(trans, to_dev(lu, "cuda"), n, ld, to_dev(piv, "cuda"), B, nrhs, ld)
        assert_bitwise(to_host(B), want, f"n={n} nrhs={nrhs} {trans}")


@pytest.mark.parametrize("n", [129, 144, 160, 161, 191, 192, 193, 224, 255, 256])
def test_getrs_block_edges(handle, n):
    """The register solve (getrs_block.cu): panel and tile edges, column counts around 4, 16 and a CTA's 64, odd
    strides, invalid pivots, a zero on the diagonal, infinities and NaN."""
    rng = np.random.default_rng(n)
    for nrhs, batch, pad in ((1, 460, 0), (4, 460, 1), (5, 460, 4), (16, 3, 0), (17, 160, 0), (70, 60, 3)):
        ld = n + pad
        lu = rng.standard_normal((batch, n, ld)).astype(np.float32)
        lu[:, np.arange(n), np.arange(n)] += 12
        piv = (np.arange(1, n + 1) + rng.integers(0, n - np.arange(n), (batch, n))).astype(np.int32)
        piv[0, 0] = 0
        piv[0, n - 1] = n + 7
        if batch > 1:
            lu[1, n // 2, n // 2] = 0.0
        b = rng.standard_normal((batch, nrhs, ld)).astype(np.float32)
        if nrhs > 2:
            b[batch - 1, 1, n - 1] = np.inf
            b[batch - 1, 2, 0] = np.nan
        want = b.copy()
        with np.errstate(all="ignore"):
            O.port_getrs("N", lu, n, ld, piv, want, nrhs, ld)
        B = to_dev(b, "cuda")
        handle.getrs("N", to_dev(lu, "cuda"), n, ld, to_dev(piv, "cuda"), B, nrhs, ld)
        assert_bitwise(to_host(B), want, f"n={n} nrhs={nrhs}")
