"""Solves with many right-hand sides. aclblasSgetrsBatched, trans N, 32 < n <= 128 with at least 65536 of them in
the batch: bit for bit against the oracle, for a packed 16-byte-aligned layout and a padded odd leading
dimension, with some matrices skipped through a NULL right-hand-side pointer. Refinements and plans with more
columns than one grid, or one pass of the generic solve, takes."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import to_dev, to_host
from test_lu_gpu import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs,batch,pad", [(64, 8, 8192, 0), (33, 1, 65536, 0), (100, 2, 32768, 3),
                                              (128, 4, 16384, 0)])
def test_getrs_many_rhs_trans_n(handle, n, nrhs, batch, pad):
    import torch

    lda = ldb = n + pad
    rng = np.random.default_rng(n * 7 + nrhs)
    a = rng.standard_normal((batch, n, lda)).astype(np.float32)
    lu = a.copy()
    piv, _, _ = O.port_getrf(lu, n, lda)
    b = rng.standard_normal((batch, nrhs, ldb)).astype(np.float32)
    want = b.copy()
    O.port_getrs("N", lu, n, lda, piv, want, nrhs, ldb)
    LU, B = to_dev(lu, "cuda"), to_dev(b, "cuda")
    bptr = torch.arange(batch, device="cuda", dtype=torch.int64) * (nrhs * ldb * 4) + B.data_ptr()
    skip = torch.arange(0, batch, 97, device="cuda")
    bptr[skip] = 0  # NULL right-hand side: the matrix is skipped
    handle.getrs("N", LU, n, lda, to_dev(piv, "cuda"), B, nrhs, ldb, bptr=bptr)
    torch.cuda.synchronize()
    got = to_host(B)
    keep = np.ones(batch, bool)
    keep[np.arange(0, batch, 97)] = False
    assert_bitwise(got[keep], want[keep], f"n={n} nrhs={nrhs}")
    assert np.array_equal(got[~keep], b[~keep])


def test_refine_more_columns_than_one_grid_takes(ob, cuda):
    """n <= 128: the solve's blocks of right-hand sides are a grid's second dimension (65535 of them at most)."""
    import torch

    n, k = 33, 64
    nrhs = (65536 * 128 // k + 1) * k
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(1, n, n, device="cuda", generator=g) + 12 * torch.eye(n, device="cuda")
    B = torch.randn(k, n, device="cuda", generator=g).repeat(nrhs // k, 1).reshape(1, nrhs, n)
    few = B[:, :k].clone()
    with ob.Handle() as h:  # its own: the workspace of this call is a gigabyte
        X, LU, piv, info, _, _ = h.refine(A, B, n, nrhs, max_iter=0, compute=ob.COMPUTE_32F)
        h.getrs("N", LU, n, n, piv, few, k, n)
        torch.cuda.synchronize()
    assert int(info[0]) == 0
    assert torch.equal(X.reshape(nrhs // k, k, n), few.expand(nrhs // k, k, n))


def test_grouped_more_columns_than_one_grid_takes(ob, handle):
    """128 < n <= 256, as above through a plan (whose groups above 128 run on the batched kernels)."""
    import torch

    n, k = 129, 64
    nrhs = 65536 * 64 + k
    g = torch.Generator(device="cuda").manual_seed(2)
    A = torch.randn(1, n, n, device="cuda", generator=g) + 24 * torch.eye(n, device="cuda")
    B = torch.randn(k, n, device="cuda", generator=g).repeat(nrhs // k, 1).reshape(1, nrhs, n)
    few = B[:, :k].clone()
    LU = A.clone()
    piv, _ = handle.getrf(LU, n, n)
    handle.getrs("N", LU, n, n, piv, few, k, n)
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.empty(1, dtype=torch.int32, device="cuda")
    with_plan = ob.GroupedPlan(handle, [n], [nrhs], [1])
    with_plan.run(handle, ob.ptr_array(A), piv, info, ob.ptr_array(B))
    torch.cuda.synchronize()
    with_plan.close()
    assert int(info[0]) == 0
    assert torch.equal(B.reshape(nrhs // k, k, n), few.expand(nrhs // k, k, n))


def test_grouped_more_columns_than_a_generic_pass(ob, handle):
    """Orders whose right-hand sides no longer fit shared memory: the generic solve's 256 columns a pass. A plan takes
    any number of them (aclblasSgetrsBatched at most 256)."""
    import torch

    n, nrhs = 2720, 300
    g = torch.Generator(device="cuda").manual_seed(3)
    A = torch.randn(1, n, n, device="cuda", generator=g) + 100 * torch.eye(n, device="cuda")
    B = torch.randn(1, nrhs, n, device="cuda", generator=g)
    LU = A.clone()
    piv, _ = handle.getrf(LU, n, n)
    want = []
    for part in (B[:, :200].clone(), B[:, 200:].clone()):
        handle.getrs("N", LU, n, n, piv, part, part.shape[1], n)
        want.append(part)
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.empty(1, dtype=torch.int32, device="cuda")
    plan = ob.GroupedPlan(handle, [n], [nrhs], [1])
    plan.run(handle, ob.ptr_array(A), piv, info, ob.ptr_array(B))
    torch.cuda.synchronize()
    plan.close()
    assert int(info[0]) == 0
    assert torch.equal(B, torch.cat(want, 1))
