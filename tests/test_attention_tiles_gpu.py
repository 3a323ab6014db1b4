"""The tiled float32 attention of prompt portions against the softmax formulas in 64 bits, at the edges of its tiles.

A score is a sum of at most 128 products, an output one of at most 1,300: 2^-24 times the square root of that, with the
exponential's own two units, stays below 2.5e-6 of the result's norm."""

from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import make_cache, step_of

pytestmark = pytest.mark.gpu

BOUND = 2.5e-6


def exact(q, kv, lengths, pasts, heads, kv_heads, dim, scale, window, chunk, keep_first, softcap, sink):
    out, at = [], 0
    for i in sorted(range(len(lengths)), key=lambda i: (lengths[i] != 1, i)):
        n, past = lengths[i], pasts[i]
        key = torch.arange(n + past, device="cuda")
        page, slot = kv.block_table[i].long()[key // kv.page_size], key % kv.page_size
        keys, values = (x[page, :, slot].double().repeat_interleave(heads // kv_heads, 1) for x in (kv.k, kv.v))
        score = torch.einsum("thd,jhd->htj", q[at : at + n].view(n, heads, dim).double(), keys) * scale
        at += n
        if softcap:
            score = softcap * torch.tanh(score / softcap)
        position = torch.arange(past, past + n, device="cuda")[:, None]
        first = torch.zeros_like(position)
        if window:
            first = torch.maximum(first, position - window + 1)
        if chunk:
            first = torch.maximum(first, position // chunk * chunk)
        seen = (key <= position) & ((key >= first) | (key < keep_first))
        score = score.masked_fill(~seen, -float("inf"))
        if sink is not None:
            score = torch.cat([score, sink.double()[:, None, None].expand(-1, n, 1)], -1)
        out.append(torch.einsum("htj,jhd->thd", torch.softmax(score, -1)[..., : n + past], values).reshape(n, -1))
    return torch.cat(out)


@pytest.mark.parametrize(
    "lengths,pasts,heads,kv_heads,dim,value_dim,extra",
    [
        ([200], [0], 4, 2, 128, 128, {}),
        ([65, 1, 130, 32], [33, 70, 200, 0], 4, 2, 64, 64, {}),
        ([33, 2], [5, 1200], 2, 1, 32, 32, {}),
        ([70], [150], 4, 4, 96, 128, {"sink": True}),
        ([129, 40], [300, 10], 4, 2, 128, 64, {"window": 50, "keep_first": 7}),
        ([100], [100], 4, 2, 64, 64, {"chunk": 37, "softcap": 5.0}),
        ([64], [1000], 2, 2, 20, 12, {"window": 300, "keep_first": 70, "sink": True}),
        ([31], [64], 2, 1, 100, 100, {"window": 1}),
        ([5, 1], [64, 9], 2, 1, 24, 24, {}),  # a single token of a size without a decode kernel
    ],
)
def test_tiles_against_the_formulas(lengths, pasts, heads, kv_heads, dim, value_dim, extra):
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.float32, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(11)
    page, width = 16, max(-(-(n + p) // 16) for n, p in zip(lengths, pasts))
    kv = make_cache(torch.float32, len(lengths) * width, kv_heads, page, dim, len(lengths), width)
    if value_dim != dim:
        kv.v = torch.randn(*kv.k.shape[:3], value_dim, generator=generator, device="cuda")
    step = step_of(lengths, pasts, list(range(len(lengths))))
    q = torch.randn(step.num_tokens, heads * dim, generator=generator, device="cuda")
    sink = torch.randn(heads, generator=generator, device="cuda") if extra.get("sink") else None
    window, chunk = extra.get("window"), extra.get("chunk")
    keep_first, softcap = extra.get("keep_first", 0), extra.get("softcap", 0.0)
    out = torch.full((step.num_tokens, heads * value_dim), float("nan"), device="cuda")
    ks.attention(q, out, step, kv, heads, kv_heads, dim, window, dim**-0.5, chunk, keep_first, softcap, sink)
    ks.check_errors()
    assert ks.kernel_counts.get("attention_tiles")
    want = exact(q, kv, lengths, pasts, heads, kv_heads, dim, dim**-0.5, window, chunk, keep_first, softcap, sink)
    error = float((out.double() - want).norm() / want.norm())
    assert error <= BOUND, f"off by {error:.2e}"


def test_a_missing_page_is_reported_and_its_keys_skipped():
    from distie_b200.kernels import make_kernels
    from distie_b200.kernels.library import KernelError

    ks = make_kernels(torch.float32, "cuda:0")
    kv = make_cache(torch.float32, 8, 1, 16, 64, 1, 8)
    kv.block_table[0, 1] = -1
    step = step_of([40], [60], [0])
    q, out = torch.randn(40, 64, device="cuda"), torch.empty(40, 64, device="cuda")
    ks.attention(q, out, step, kv, 1, 1, 64, None, 0.125)
    with pytest.raises(KernelError):
        ks.check_errors()
    assert torch.isfinite(out).all()
    ks.attention(q, out, step, kv, 1, 1, 64, 8, 0.125)  # the page lies before every row's window
    ks.check_errors()


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where,window,keep_first", [(150, None, 0), (70, 40, 0), (3, 40, 5), (2, 40, 2), (99, 1, 0)])
def test_a_value_that_is_not_finite_reaches_the_tokens_that_see_it_alone(where, window, keep_first, bad):
    """The key's tile holds rows before it, behind it and, with a window, past it; the first keys are kept for good or not."""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.float32, "cuda:0")
    past, n, heads, dim = 60, 130, 2, 64
    kv = make_cache(torch.float32, 16, 1, 16, dim, 1, 16)
    step = step_of([n], [past], [0])
    generator = torch.Generator(device="cuda").manual_seed(4)
    q = torch.randn(n, heads * dim, generator=generator, device="cuda")
    page, slot = kv.block_table[0].long()[where // 16], where % 16
    kv.v[page, 0, slot] = 0.0
    want = exact(q, kv, [n], [past], heads, 1, dim, 0.125, window, None, keep_first, 0.0, None)
    kv.v[page, 0, slot, 5] = bad
    out = torch.empty(n, heads * dim, device="cuda")
    ks.attention(q, out, step, kv, heads, 1, dim, window, 0.125, None, keep_first)
    ks.check_errors()
    assert ks.kernel_counts.get("attention_tiles")
    position = torch.arange(past, past + n, device="cuda")
    sees = (position >= where) & ((position - where < (window or 10**6)) | (where < keep_first))
    spoiled = torch.zeros(n, heads, dim, dtype=torch.bool, device="cuda")
    spoiled[sees, :, 5] = True
    spoiled = spoiled.view(n, -1)
    assert torch.equal(~torch.isfinite(out), spoiled)
    error = float((out.double() - want)[~spoiled].norm() / want[~spoiled].norm())
    assert error <= BOUND, f"off by {error:.2e}"


def test_a_key_that_is_not_finite_reaches_the_tokens_that_see_it_alone():
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.float32, "cuda:0")
    kv = make_cache(torch.float32, 8, 1, 16, 64, 1, 8)
    step = step_of([100], [20], [0])
    q, out, clean = (torch.randn(100, 64, generator=torch.Generator(device="cuda").manual_seed(5 + i), device="cuda") for i in range(3))
    ks.attention(q, clean, step, kv, 1, 1, 64, None, 0.125)
    kv.k[kv.block_table[0].long()[80 // 16], 0, 80 % 16, 3] = float("nan")
    ks.attention(q, out, step, kv, 1, 1, 64, None, 0.125)
    assert torch.equal(out[:60], clean[:60]) and not torch.isfinite(out[60:]).any()
