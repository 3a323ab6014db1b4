"""Routed products on pairs of CTAs with tiles of 256 rows: the same numbers as with tiles of 128, bit by bit."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,ff,counts", [
    (136, 72, [0, 1, 127, 128, 129, 255, 256, 257, 0, 513]), (512, 768, [700, 0, 0, 300]), (1536, 2240, [188] * 16), (64, 8, [600]),
])
@pytest.mark.parametrize("act", [None, "gelu"])
def test_tiles_of_256_rows_equal_tiles_of_128(monkeypatch, hidden, ff, counts, act):
    from distie_b200.kernels import device, make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    g = torch.Generator(device="cuda").manual_seed(hidden + len(counts))
    experts, tokens = len(counts), sum(counts)
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])
    ids = ids[torch.randperm(tokens, generator=torch.Generator().manual_seed(1))].cuda()[:, None].contiguous()
    weights = torch.rand(tokens, 1, generator=g, device="cuda") + 0.1
    x = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16)
    make = lambda *shape: (torch.randn(*shape, generator=g, device="cuda") / shape[-1] ** 0.5).to(torch.bfloat16)  # noqa: E731
    up, down = make(experts, ff * (2 if act is None else 1), hidden), make(experts, hidden, ff)
    got = []
    for tile in (128, 256):
        monkeypatch.setattr(device, "grouped_tile", lambda *args: tile)
        before = ks.kernel_counts.get("gemm_tcgen05_grouped", 0)
        got.append(ks.routed_swiglu(x, ids, weights, up, down) if act is None else ks.routed_act(x, ids, weights, up, down, act))
        ks.check_errors()
        assert ks.kernel_counts["gemm_tcgen05_grouped"] == before + 1
    assert torch.equal(got[0], got[1]) and bool(torch.isfinite(got[0]).all()) and float(got[0].abs().max()) > 0


@pytest.mark.parametrize("top,scale_input,limit,identity", [(3, True, None, 0), (2, False, 0.5, 0), (4, False, None, 3), (3, False, 1.0, 1)])
def test_tiles_of_256_rows_with_every_option(monkeypatch, top, scale_input, limit, identity):
    """Several experts a token, weights on either side, capped gates, experts that return their input: as in tiles of 128, bit
    by bit, and as the formulas have it."""
    import ref_kernels as ref
    from distie_b200.kernels import device, make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    g = torch.Generator(device="cuda").manual_seed(top)
    tokens, experts, hidden, ff = 300, 5, 136, 72
    ids = torch.rand(tokens, experts + identity, generator=g, device="cuda").topk(top, dim=1).indices.int().contiguous()
    weights = torch.rand(tokens, top, generator=g, device="cuda") + 0.1
    x = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16)
    up, down = ((torch.randn(*shape, generator=g, device="cuda") / shape[-1] ** 0.5).to(torch.bfloat16)
                for shape in ((experts, 2 * ff, hidden), (experts, hidden, ff)))
    got = []
    for tile in (128, 256):
        monkeypatch.setattr(device, "grouped_tile", lambda *args: tile)
        before = ks.kernel_counts.get("gemm_tcgen05_grouped", 0)
        got.append(ks.routed_swiglu(x, ids, weights, up, down, scale_input, limit, identity))
        ks.check_errors()
        assert ks.kernel_counts["gemm_tcgen05_grouped"] == before + 1
    assert torch.equal(got[0], got[1])
    want = ref.routed_swiglu(x.cpu(), ids.cpu(), weights.cpu(), up.cpu(), down.cpu(), scale_input, limit, identity).cuda()
    assert float((got[1] - want).norm() / want.norm()) < 1e-2  # (inputs and the hidden layer rounded to bfloat16)
