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
    if k >= 1024 and m >= 128:  # (of a few rows the library cuts K, which is nearer than FMA all along it)
        fma = torch.nn.functional.linear(x, w, b)
        assert float((got.double() - want).norm()) < float((fma.double() - want).norm())
        assert float((got.double() - want).norm() / want.norm()) < 2.5e-7  # (1.4e-7 at K 1,536, 1.9e-7 at 9,000)


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


@pytest.mark.parametrize("k", [96, 768, 776, 1544, 6152])  # one, two and eight warps a row, rows read twice
def test_rows_of_the_smallest_and_largest_numbers_keep_their_bits(ks, k):
    """Every float32 number has three planes, whatever its size: rows and columns of 2^-149 to 2^127 against 64 bits, as near
    to them as ordinary ones are (their own last bits are what a row below 2^-126 holds of them)."""
    g = torch.Generator(device="cuda").manual_seed(k)
    sizes = torch.tensor([-149, -140, -126, -120, -116, -112, -100, -64, -41, -40, -39, 0, 30, 39, 40, 41, 64, 100, 126], device="cuda")
    x = torch.rand(3 * sizes.numel(), k, generator=g, device="cuda") * 2 - 1
    w = torch.rand(4 * sizes.numel(), k, generator=g, device="cuda") * 2 - 1
    x = torch.ldexp(x, sizes.repeat(3)[:, None])
    w = torch.ldexp(w, sizes.repeat_interleave(4)[:, None])
    x[:, 5] = torch.where(x.abs().amax(1) == 0, 2.0**-149, x[:, 5])
    want = x.double() @ w.double().t()
    got = product(ks, x, w).double()
    scale = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)
    inside = (want.abs() < 3.4e38) & (scale > 0)
    bound = (8 + (k / 128) ** 0.5) * 2.0**-24 * scale + 2.0**-149
    assert bool(((got - want).abs() <= bound)[inside].all()), float(((got - want).abs() / bound)[inside].max())
    beyond = want.abs() > 3.5e38
    assert torch.equal(got[beyond], want[beyond].sign() * float("inf"))


def test_infinity_times_the_smallest_numbers_is_infinity(ks):
    x, w = torch.ones(200, 64, device="cuda"), torch.ones(128, 64, device="cuda")
    x[3, 9], w[4, 9], w[5, 9], w[6, 9] = float("inf"), 2.0**-149, -(2.0**-140), 0.0
    w[7] *= 2.0**127
    w[7, 9] = -(2.0**-149)
    got = product(ks, x, w)
    assert got[3, 4] == float("inf") and got[3, 5] == float("-inf") and bool(got[3, 6].isnan()) and got[3, 7] == float("-inf")
    assert bool(torch.isfinite(got[:3, :7]).all()) and bool(torch.isfinite(got[4:, :7]).all())


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3e38])
def test_rows_that_are_not_finite_take_no_longer(ks, value):
    x, w = torch.randn(777, 1536, device="cuda"), torch.randn(2048, 1536, device="cuda")
    odd = x.clone()
    odd[::7, 100] = value

    def time(x):
        best = 1e9
        for _ in range(10):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            product(ks, x, w)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        return best

    time(x)
    assert time(odd) < 2 * time(x)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_kernel_is_loaded_with_the_kernel_set(monkeypatch, dtype):
    """Not by the first large product, which would wait for the compiler where the unit was not built ahead."""
    from distie_b200.kernels import library, make_kernels

    seen, load = [], library.load_unit
    monkeypatch.setattr(library, "load_unit", lambda unit: seen.append(unit) or load(unit))
    make_kernels(dtype, "cuda:0")
    assert "float32" in seen
