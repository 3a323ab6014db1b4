"""Products of few columns whose reduction is split over pairs of CTAs, against the product in 64 bits.

The operands are bfloat16 and the sums float32: K additions of 2^-24 each in a chain are at most sqrt(K) * 2^-23 of the
result's norm, and truncating accumulators K / 16 * 2^-24 more."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(256, 1, 704), (257, 16, 1536), (1001, 128, 3080), (2048, 130, 1000), (640, 250, 4088), (511, 96, 776)])
def test_slices_add_up_to_the_product(m, n, k):
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(m, k, generator=generator, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=generator, device="cuda") / k**0.5).to(torch.bfloat16)
    slices = ks.linear_split(x, w)
    ks.check_errors()
    assert "gemm_tcgen05_split" in ks.kernel_counts and slices.shape[0] > 1 and slices.shape[1:] == (m, n)
    want = x.double() @ w.double().t()
    error = float((slices.double().sum(0) - want).norm() / want.norm())
    assert error <= k**0.5 * 2**-23 + k / 16 * 2**-24, f"off by {error:.2e}"


def test_the_router_against_the_product_in_64_bits():
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(700, 1536, generator=generator, device="cuda").to(torch.bfloat16)
    router = (torch.randn(24, 1536, generator=generator, device="cuda") / 40).to(torch.bfloat16)
    ids, weights = ks.route_top(x, router, 3)
    score = torch.sigmoid(x.double() @ router.double().t())
    top, want = score.topk(4, -1)
    clear = (top[:, :3] - top[:, 1:] > 1e-5).all(-1)
    assert int(clear.sum()) > 650 and torch.equal(ids[clear].long(), want[clear, :3])
    assert float((weights.double() - top[:, :3])[clear].abs().max()) < 1e-5


@pytest.mark.parametrize("experts,width", [(16, 1536), (256, 1024), (64, 3584)])
def test_a_token_is_routed_alike_in_every_step(experts, width):
    """Chosen experts are whole numbers: a token's must not hang on how many tokens share its step.  (The logits are one
    product in one order of summation from 256 rows on; 6,000 rows are more tiles than any split takes.)"""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(6000, width, generator=generator, device="cuda").to(torch.bfloat16)
    router = (torch.randn(experts, width, generator=generator, device="cuda") / width**0.5).to(torch.bfloat16)
    ids, weights = ks.route_top(x, router, 3)
    for rows in (300, 1001, 2048):
        few_ids, few_weights = ks.route_top(x[:rows], router, 3)
        assert torch.equal(few_ids, ids[:rows]) and torch.equal(few_weights, weights[:rows])
