"""Attention of prompt portions with two query tiles a CTA and keys cut into shares, against the formulas in float32.

Groups that pair up and groups that do not, tiles without a partner, units cut into pieces and rows of units cut into
shares, partial tiles, every mask and score option, heads that fill no tile, pages of every size, scores that rise by
more than the range in which exponentials are taken without a new maximum."""

from __future__ import annotations

import pytest
import torch

import ref_kernels as ref
from test_kernels_gpu import close, filled_cache_for, step_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ks():
    from distie_b200.kernels import make_kernels

    return make_kernels(torch.bfloat16, "cuda:0")


def in_pairs(ks, monkeypatch, *args):
    """The kernel of pairs, whatever the rule would take: it has to be the one that runs."""
    from distie_b200.kernels import device

    before = ks.kernel_counts.get("attention_prefill_pairs", 0)
    with monkeypatch.context() as forced:
        forced.setattr(device.DeviceKernels, "_in_pairs", lambda *args: True)
        ks.attention(*args)
    ks.check_errors()
    assert ks.kernel_counts["attention_prefill_pairs"] == before + 1


def run(ks, monkeypatch, heads, kv_heads, head_dim, value_dim, page, tokens, pasts, window=None, chunk=None, keep_first=0, softcap=0.0,
        sink=False, scale=None, keys=None, missing=None):
    from distie_b200.kernels.interface import KvSlot

    g = torch.Generator(device="cuda").manual_seed(heads * 31 + head_dim + sum(tokens))
    kv = filled_cache_for(torch.bfloat16, kv_heads, head_dim, page, [p + n for p, n in zip(pasts, tokens)])
    values = torch.randn(*kv.k.shape[:3], value_dim, generator=g, device="cuda").to(torch.bfloat16)
    kv = KvSlot(kv.k, values, kv.block_table, page, kv.num_pages)
    if keys is not None:
        keys(kv)
    step = step_of(tokens, pasts, list(range(len(tokens))))
    q = torch.randn(step.num_tokens, heads * head_dim, generator=g, device="cuda").to(torch.bfloat16)
    sinks = torch.randn(heads, generator=g, device="cuda") if sink else None
    out = torch.full((step.num_tokens, heads * value_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    args = (heads, kv_heads, head_dim, window, scale or head_dim**-0.5, chunk, keep_first, softcap, sinks)
    want = ref.attention(q, step, kv, *args)
    if missing is not None:
        missing(kv)
    in_pairs(ks, monkeypatch, q, out, step, kv, *args)
    close(out, want, torch.bfloat16, f"{heads} heads, {tokens} behind {pasts}")


@pytest.mark.parametrize("heads,kv_heads", [(4, 2), (6, 2), (7, 1), (3, 3), (1, 1), (40, 8)])
@pytest.mark.parametrize("tokens,pasts", [
    ([2], [0]), ([128], [0]), ([129], [0]), ([257], [3]), ([300, 2, 128, 511], [900, 4000, 0, 1]), ([150], [5000]), ([1, 1, 700], [30, 2000, 1500]),
])
def test_units_pieces_and_shares(ks, monkeypatch, heads, kv_heads, tokens, pasts):
    run(ks, monkeypatch, heads, kv_heads, 128, 128, 16, tokens, pasts)


def test_more_tiles_than_lanes_and_units_than_shares(ks, monkeypatch):
    run(ks, monkeypatch, 6, 2, 64, 64, 16, [2 + 5 * i for i in range(70)], [37 * (i % 9) for i in range(70)])
    run(ks, monkeypatch, 14, 2, 128, 128, 16, [260] * 9 + [1300], [1000] * 9 + [2100])


@pytest.mark.parametrize("head_dim,value_dim,page,window,chunk,keep_first,softcap,sink", [
    (128, 128, 8, 300, None, 0, 0.0, False), (64, 64, 128, 1000, None, 40, 0.0, True), (128, 128, 32, None, 500, 0, 0.0, False),
    (96, 96, 16, 64, None, 200, 0.0, False), (128, 64, 16, None, None, 0, 5.0, True), (64, 128, 64, 200, None, 3, 2.5, False),
    (40, 8, 16, None, 128, 0, 0.0, True), (88, 120, 16, 1, None, 0, 0.0, False),
])
@pytest.mark.parametrize("heads,kv_heads", [(6, 3), (5, 1)])
def test_masks_caps_sinks_and_sizes(ks, monkeypatch, heads, kv_heads, head_dim, value_dim, page, window, chunk, keep_first, softcap, sink):
    run(ks, monkeypatch, heads, kv_heads, head_dim, value_dim, page, [1, 333, 2, 140], [10, 1700, 900, 0], window, chunk, keep_first, softcap, sink)


@pytest.mark.parametrize("kv_heads", [1, 2])
def test_pages_that_a_window_gave_back_are_not_asked_for(ks, monkeypatch, kv_heads):
    pasts, window = [2000, 650], 300

    def missing(kv):
        for seat, past in enumerate(pasts):
            kv.block_table[seat, : max(0, past - window + 1) // 16] = -1

    run(ks, monkeypatch, 2, kv_heads, 128, 128, 16, [300, 290], pasts, window, missing=missing)


@pytest.mark.parametrize("factor,scale", [(1.0, 3.0), (4.0, 2.0)])
def test_scores_that_leave_the_range(ks, monkeypatch, factor, scale):
    """Keys grow along the request: a row's scores rise by hundreds in base-2 units, past 2^30 many times over."""
    def keys(kv):
        growth = torch.linspace(0.01, factor, kv.block_table.shape[1], device="cuda")
        for seat in range(kv.block_table.shape[0]):
            row = kv.block_table[seat]
            held = row[row >= 0].long()
            kv.k[held] = (kv.k[held].float() * growth[: held.numel(), None, None, None]).to(torch.bfloat16)

    run(ks, monkeypatch, 4, 2, 128, 128, 16, [200, 150], [1800, 300], scale=scale, keys=keys)


@pytest.mark.parametrize("past", [700, 1500])  # a tile by itself, and one whose keys are cut into pieces
@pytest.mark.parametrize("low,high", [(15.0, 22.0), (34.0, 60.0)])  # base-2 units: without and with a new maximum
def test_weights_above_the_maximum_in_use_count_as_they_are_rounded(ks, monkeypatch, past, low, high):
    """Sixteen keys' scores lie `low` to `high` base-2 units above all before them; their weights, rounded to bfloat16, have to
    count in the row's sum as they count in the product.  An output is then off along its own direction by no more than its
    own rounding (2^-9 at most, 1.1e-3 in the root mean square, of each of 128 elements whose squares weigh as normal numbers' do:
    1.1e-3 (3 / 128)^1/2 = 1.7e-4) and what the other keys' share of 1500 / 2^19 leaves; with weights summed before they are
    rounded, by up to 2^-9 at once."""
    g = torch.Generator(device="cuda").manual_seed(past)
    heads, tokens, at, scale = 4, 200, 32, 128**-0.5  # (keys 512 to 527)
    kv = filled_cache_for(torch.bfloat16, 2, 128, 16, [past + tokens])
    kv.k.zero_()
    kv.k[int(kv.block_table[0, at]), :, :, 0] = 16.0
    step = step_of([tokens], [past], [0])
    q = torch.zeros(tokens, heads, 128, device="cuda")
    q[..., 0] = torch.empty(tokens, heads, device="cuda").uniform_(low, high, generator=g) * 0.6931 / (16 * scale)
    q = q.to(torch.bfloat16)
    out = torch.empty(tokens, heads * 128, dtype=torch.bfloat16, device="cuda")
    in_pairs(ks, monkeypatch, q.reshape(tokens, -1), out, step, kv, heads, 2, 128, None, scale)
    keys = torch.arange(past + tokens, device="cuda")
    pages = kv.block_table[0, keys // 16].long()
    k, v = (c[pages, :, keys % 16].double().repeat_interleave(heads // 2, dim=1) for c in (kv.k, kv.v))
    scores = torch.einsum("thd,nhd->thn", q.double(), k) * scale
    scores.masked_fill_(keys[None, None] > step.positions.long()[:, None, None], float("-inf"))
    want = torch.einsum("thn,nhd->thd", scores.softmax(-1), v)
    along = (out.double().reshape_as(want) * want).sum(-1) / (want * want).sum(-1) - 1
    assert float(along.square().mean().sqrt()) < 3e-4


@pytest.mark.parametrize("past,tokens,window,keep_first,at,free", [
    (0, 200, None, 0, 190, slice(0, 128)), (70, 300, None, 0, 330, slice(0, 128)), (70, 300, None, 0, 260, slice(0, 128)),
    (4990, 200, None, 0, 5150, slice(0, 128)),  # (cut: a piece may end with blocks that the first tile does not see)
    (100, 256, 100, 0, 50, slice(128, 256)), (100, 256, None, 0, 50, slice(0, 0)), (3000, 256, 100, 0, 2930, slice(128, 256)),
    (3000, 256, 100, 200, 2930, slice(128, 256)), (100, 256, 30, 40, 100, slice(0, 0)), (300, 256, 100, 129, 230, slice(0, 0)),
    (600, 256, 300, 400, 390, slice(0, 0)), (650, 256, 100, 300, 560, slice(128, 256)),
])
@pytest.mark.parametrize("heads", [1, 7])
def test_a_value_that_is_not_finite_stays_with_the_tiles_that_see_its_block(ks, monkeypatch, heads, past, tokens, window, keep_first, at, free):
    """Two tiles of one request share a unit; blocks of keys that only one of them sees leave the other one's rows alone."""
    kv = filled_cache_for(torch.bfloat16, 1, 128, 16, [past + tokens])
    step = step_of([tokens], [past], [0])
    q = torch.randn(tokens, heads * 128, device="cuda").to(torch.bfloat16)
    args = (heads, 1, 128, window, 128**-0.5, None, keep_first)
    want = ref.attention(q, step, kv, *args)
    kv.v[int(kv.block_table[0, at // 16]), :, at % 16] = float("nan")
    out = torch.zeros_like(q)
    in_pairs(ks, monkeypatch, q, out, step, kv, *args)
    if out[free].numel():
        close(out[free], want[free], torch.bfloat16)
    sees = torch.arange(past, past + tokens, device="cuda")
    sees = (sees >= at) & ((sees - at < (window or 1 << 30)) | (at < keep_first))
    assert bool(out[sees].isnan().all())


@pytest.mark.parametrize("past,missing", [(1300, 40), (1300, 93), (300, 0)])  # in parts of cut units, in a whole one
def test_a_missing_page_sets_the_error_word(ks, monkeypatch, past, missing):
    from distie_b200.kernels.library import KernelError

    kv = filled_cache_for(torch.bfloat16, 2, 128, 16, [past + 200])
    step = step_of([200], [past], [0])
    q = torch.randn(200, 4 * 128, device="cuda").to(torch.bfloat16)
    page, kv.block_table[0, missing] = int(kv.block_table[0, missing]), -1
    with pytest.raises(KernelError, match="portion of a prompt"):
        in_pairs(ks, monkeypatch, q, torch.empty_like(q), step, kv, 4, 2, 128, None, 128**-0.5)
    kv.block_table[0, missing] = page  # and the next call is as if nothing had been
    out = torch.full_like(q, float("nan"))
    in_pairs(ks, monkeypatch, q, out, step, kv, 4, 2, 128, None, 128**-0.5)
    close(out, ref.attention(q, step, kv, 4, 2, 128, None, 128**-0.5), torch.bfloat16, "after a missing page")


def test_steps_that_the_rule_sends_to_either_kernel_count_apart(ks):
    kv = filled_cache_for(torch.bfloat16, 2, 128, 16, [4130])
    for tokens, past, pairs in ((130, 0, 0), (130, 4000, 1)):
        step = step_of([tokens], [past], [0])
        q = torch.randn(tokens, 12 * 128, device="cuda").to(torch.bfloat16)
        before = [ks.kernel_counts.get(name, 0) for name in ("attention_prefill_tcgen05", "attention_prefill_pairs")]
        ks.attention(q, torch.empty_like(q), step, kv, 12, 2, 128, None, 128**-0.5)
        ks.check_errors()
        after = [ks.kernel_counts.get(name, 0) for name in ("attention_prefill_tcgen05", "attention_prefill_pairs")]
        assert [b - a for a, b in zip(before, after)] == [1, pairs]
