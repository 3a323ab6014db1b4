"""The RMS norm in the reference's order behind a sum of terms, which is float32 in every engine."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hidden", [64, 50, 1536])  # a width that the kernel over slices refuses among them
@pytest.mark.parametrize("rows", [None, [4, 0]])
def test_a_norm_adds_terms_in_float32(dtype, hidden, rows):
    from distie_b200.kernels import make_kernels
    from distie_b200.kernels.interface import Terms
    from distie_b200.parts.norm import RMSNorm

    ks = make_kernels(dtype, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(hidden)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    residual, weight, slices, plain = normal(5, hidden), normal(hidden), normal(3, 5, hidden), normal(5, hidden).to(dtype)
    index = None if rows is None else torch.tensor(rows, dtype=torch.int32, device="cuda")
    want = residual.double() + 0.5 * slices.double().sum(0) + 2.0 * plain.double()
    held = residual.clone()
    out = torch.empty(5 if rows is None else len(rows), hidden, dtype=dtype, device="cuda")
    RMSNorm(weight, 1e-6, ks).apply(Terms([(slices, 0.5), (plain, 2.0)]), held, out, index)
    if rows is not None:
        want = want[index.long()]
    else:  # the sum of at most five float32 numbers
        assert float((held.double() - want).abs().max()) <= 5 * 2**-24 * 8
    unit = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6) * weight.double()
    # float32: rounding of the sums and the square root; bfloat16: of the norm and of its product with the weight
    bound = 1e-6 if dtype == torch.float32 else 2**-8
    assert float((out.double() - unit).norm() / unit.norm()) <= bound


def test_a_sum_of_another_type_is_refused():
    from distie_b200.kernels import make_kernels
    from distie_b200.kernels.library import KernelError

    ks = make_kernels(torch.float32, "cuda:0")
    residual, out = torch.zeros(2, 64, device="cuda"), torch.empty(2, 64, device="cuda")
    with pytest.raises(KernelError):
        ks.add_rmsnorm(torch.zeros(2, 64, dtype=torch.bfloat16, device="cuda"), residual, torch.ones(64, device="cuda"), 1e-6, out)
