"""Float32 products on the tensor cores against 64-bit values: no further from them than FMA products are."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def ks(monkeypatch):
    from distie_b200.kernels import device, make_kernels

    monkeypatch.setattr(device, "wide_pays", lambda *args: True)
    return make_kernels(torch.float32, "cuda:0")


def product(ks, x, w, bias=None):
    before = ks.kernel_counts.get("gemm_float32", 0)
    out = ks.linear(x, w, bias)
    ks.check_errors()
    assert ks.kernel_counts["gemm_float32"] == before + 1, "the kernel was meant to run"
    return out


@pytest.mark.parametrize("m,n,k,bias", [
    (1, 4, 8, False), (127, 132, 64, True), (128, 128, 128, False), (129, 60, 136, True), (300, 1000, 200, True), (5, 260, 1536, False),
    (777, 2048, 1536, True), (260, 516, 9000, False), (1030, 64, 72, True),
])
def test_products_of_ordinary_numbers(ks, m, n, k, bias):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x, w = torch.randn(m, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda") / k**0.5
    b = torch.randn(n, generator=g, device="cuda") if bias else None
    want = torch.nn.functional.linear(x.double(), w.double(), None if b is None else b.double())
    got = product(ks, x, w, b)
    # Sums of 128 terms cut off at 24 bits (eight additions of up to 2^-24 each), then rounded sums of these.
    bound = (8 + (k / 128) ** 0.5) * 2.0**-24
    assert float((got.double() - want).norm() / want.norm()) < bound
    assert float((got.double() - want).abs().max()) < 16 * bound * float(want.std())


def test_rows_of_a_wider_matrix_and_numbers_of_every_size(ks):
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(200, 640, generator=g, device="cuda")[:, 64:320]
    w = torch.randn(136, 256, generator=g, device="cuda") * torch.exp2(torch.randint(-30, 30, (136, 1), generator=g, device="cuda").float())
    x = x * 1.0
    wide = torch.zeros(200, 640, device="cuda")
    wide[:, 64:320] = x
    want = x.double() @ w.double().t()
    got = product(ks, wide[:, 64:320], w)
    assert float(((got.double() - want).abs() / (x.double().norm(dim=1)[:, None] * w.double().norm(dim=1))).max()) < 2e-6


def test_numbers_that_are_not_finite_and_the_largest(ks):
    """As the sum of products in float32 gives them: infinities stay infinite, their differences are not numbers, the largest
    numbers keep their value, and nothing spreads beyond its row and column."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w = torch.randn(150, 96, generator=g, device="cuda"), torch.randn(140, 96, generator=g, device="cuda")
    w[:, 7] = torch.where(w[:, 7].abs() < 0.1, 0.5, w[:, 7])
    w[3, 7] = 1.0  # one plane holds it, the others are zero
    x[10, 7], x[20, 7], x[30, 5] = float("inf"), float("-inf"), float("nan")
    x[40], w[50] = 0.0, 0.0
    x[40, 0], w[50, 0] = 3.4028234e38, 1.0
    x[60, 3], w[70, 3] = float("inf"), float("-inf")
    want = (x.double() @ w.double().t()).float()
    got = product(ks, x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
    keep = torch.isfinite(want)
    error = (got.double() - x.double() @ w.double().t()).abs() / (x.double().norm(dim=1)[:, None] * w.double().norm(dim=1))
    assert float(error[keep].max()) < 2e-6
    assert float(got[40, 50]) == 3.4028234663852886e38
