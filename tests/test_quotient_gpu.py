"""The multipliers of the blocked LU kernels are a / b of the device: matrices whose first column is b and smaller
a's, the rest of the identity, so that the factors' first column holds the quotients."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quotients(handle, n, b, a, pivot=True):
    """The multipliers of a (batch, n - 1) for pivots b (batch), as getrf of order n forms them."""
    import torch

    A = torch.zeros(b.shape[0], n, n, device="cuda")
    A[:, range(1, n), range(1, n)] = 1.0
    A[:, 0, 0] = b
    A[:, 0, 1:] = a
    handle.getrf(A, n, n, pivot=pivot)
    return A[:, 0, 1:]


def _numerators(g, b, count, low):
    """Magnitudes in [low, |b|]: |b| itself, its neighbours, powers of two, significands of ones, low, random."""
    import torch

    e = torch.frexp(b).exponent - 1
    spread = torch.randint(0, 60, (b.shape[0], count), device="cuda", generator=g, dtype=torch.int32)
    m = 1.0 + torch.rand(b.shape[0], count, device="cuda", generator=g)
    m[:, 0] = 1.0
    m[:, 1] = 2.0 - 2.0 ** -23
    a = torch.ldexp(m, torch.maximum(e.unsqueeze(1) - spread, torch.tensor(int(np.log2(low)), device="cuda")))
    a[:, 2] = b
    a[:, 3] = torch.nextafter(b, torch.zeros_like(b))
    a[:, 4] = torch.ldexp(torch.ones_like(b), e)
    a[:, 5] = low
    a = torch.minimum(a, b.unsqueeze(1))
    return torch.where(torch.rand(a.shape, device="cuda", generator=g) < 0.5, -a, a)


@pytest.mark.parametrize("exponent", [-60, 0, 59, 60])
def test_every_significand(handle, exponent):
    """33 <= n <= 128: every divisor of a binade; the first and last of the range that the reciprocal serves."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(exponent + 100)
    for start in range(0, 1 << 23, 1 << 17):
        s = torch.arange(start, start + (1 << 17), device="cuda", dtype=torch.int32)
        b = (s + ((exponent + 127) << 23)).view(torch.float32)
        a = _numerators(g, b, 32, 2.0 ** -60)
        got = _quotients(handle, 33, b, a)
        assert torch.equal(got.view(torch.int32), (a / b.unsqueeze(1)).view(torch.int32)), start


@pytest.mark.parametrize("n", [64, 97, 128, 129, 300])
def test_other_orders(handle, n):
    """The other kernels on the same steps: random divisors, the significand of ones and a zero among the a's."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    s = torch.randint(0, 1 << 23, (256,), device="cuda", generator=g, dtype=torch.int32)
    s[:4] = torch.tensor([0, 1, (1 << 23) - 2, (1 << 23) - 1], device="cuda")
    b = (s + (127 << 23)).view(torch.float32)
    a = _numerators(g, b, n - 1, 2.0 ** -60)
    a[:, 7] = 0.0
    a[:, 8] = -0.0
    got = _quotients(handle, n, b, a)
    assert torch.equal(got.view(torch.int32), (a / b.unsqueeze(1)).view(torch.int32))


@pytest.mark.parametrize("n", [33, 128, 129, 300])
def test_numerators_above_the_divisor(handle, n):
    """Without pivoting a may be larger than b: quotients up to 2^120, numerators beyond the range, not finite."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n + 1)
    b = torch.ldexp(1.0 + torch.rand(512, device="cuda", generator=g), torch.randint(-60, 61, (512,), device="cuda", generator=g))
    b[0], b[1], b[2], b[3] = 2.0 ** -60, 2.0 ** 60, 2.0 - 2.0 ** -23, -3.0
    shape = (512, n - 1)
    a = torch.ldexp(1.0 + torch.rand(shape, device="cuda", generator=g), torch.randint(-70, 71, shape, device="cuda", generator=g))
    a[:, 0], a[:, 1], a[:, 2], a[:, 3] = 2.0 ** 60, 2.0 ** -60, 0.0, -0.0
    a[5, 4], a[6, 5] = float("inf"), float("nan")
    want = a / b.unsqueeze(1)
    got = _quotients(handle, n, b, a, pivot=False)
    same = (got.view(torch.int32) == want.view(torch.int32)) | (got.isnan() & want.isnan())
    assert bool(same.all())
