"""Which of two kernels a step takes: the rules against steps that were timed both ways on a B200.

The lines are drawn from estimates that are within 10 % of a time, so only steps are asked for here whose two times are a
quarter and more apart."""

from __future__ import annotations

import pytest
import torch

from distie_b200.kernels import device
from distie_b200.kernels.device import chunks_pay, grouped_tile, pairs_pay, tiles_pay, wide_pays


@pytest.mark.parametrize("rule,key,value,heads,portions,tokens,walk,chunks", [
    # rule, sizes, heads, portions, tokens of each, us token by token, us in chunks
    ("delta", 16, 16, 40, 16, 155, 65.6, 247.9),
    ("delta", 32, 32, 28, 16, 155, 74.6, 210.0),
    ("delta", 64, 64, 40, 16, 155, 242.1, 398.6),
    ("delta", 64, 64, 40, 4, 158, 69.3, 114.9),
    ("delta", 128, 128, 12, 4, 64, 32.4, 49.0),
    ("delta", 128, 128, 12, 1, 2048, 507.0, 169.0),
    ("delta", 16, 16, 4, 1, 512, 83.0, 33.9),
    ("delta", 96, 96, 40, 1, 1024, 320.5, 196.4),
    ("ssd", 16, 16, 40, 16, 71, 27.8, 82.0),
    ("ssd", 32, 32, 28, 16, 72, 30.5, 65.9),
    ("ssd", 128, 128, 1, 1, 96, 20.2, 28.5),
    ("ssd", 128, 128, 12, 1, 2048, 372.0, 92.0),
    ("ssd", 128, 128, 40, 32, 64, 682.8, 314.7),
    ("gated", 16, 16, 40, 16, 71, 33.8, 82.0),
    ("gated", 32, 32, 12, 16, 80, 21.6, 36.4),
    ("ssd", 128, 128, 24, 4, 256, 180.6, 80.5),
])
def test_recurrences_run_in_chunks_where_that_is_faster(rule, key, value, heads, portions, tokens, walk, chunks):
    assert chunks_pay(rule, portions * tokens, portions, heads, key, value) == (chunks < walk)


@pytest.mark.parametrize("heads,size,portions,tokens,past,plain,tiles", [
    # heads, their size, portions, tokens of each, tokens before them, us with a block per token and head, us in tiles
    (40, 128, 32, 2, 0, 7.3, 57.9),
    (40, 128, 16, 8, 0, 14.6, 34.2),
    (40, 128, 16, 2, 70, 25.7, 57.8),
    (12, 128, 32, 2, 0, 4.5, 24.6),
    (2, 64, 16, 8, 0, 3.9, 6.9),
    (2, 16, 1, 128, 300, 72.7, 21.6),
    (28, 16, 32, 6, 128, 146.7, 37.8),
    (1, 32, 8, 4, 1000, 168.2, 45.7),
    (40, 64, 8, 24, 1000, 1466.0, 120.3),
    (12, 32, 8, 3, 300, 54.9, 27.1),
])
def test_float32_attention_runs_in_tiles_where_that_is_faster(heads, size, portions, tokens, past, plain, tiles):
    assert tiles_pay(portions * tokens, portions, tokens + past, heads, size) == (tiles < plain)


@pytest.mark.parametrize("heads,kv_heads,window,portions,one,two", [
    # heads, those of keys, window, (cached, new) tokens of the portions, us with one and with two tiles a CTA
    (12, 2, 0, [(0, 130)], 10.9, 13.4),
    (12, 2, 0, [(6000, 130)], 76.9, 36.3),
    (12, 2, 0, [(0, 1024)], 18.8, 24.9),
    (12, 2, 0, [(9000, 1000)], 123.1, 77.3),
    (28, 4, 0, [(4000, 2048)], 253.3, 160.2),
    (28, 4, 0, [(100, 2)] * 64, 99.6, 50.7),
    (40, 8, 0, [(200, 64)], 13.1, 17.7),
    (7, 1, 0, [(0, 777)], 17.5, 23.2),
    (8, 8, 0, [(0, 128)] * 16, 9.2, 12.8),
])
def test_prompt_attention_takes_two_tiles_a_cta_where_that_is_faster(heads, kv_heads, window, portions, one, two):
    assert pairs_pay(portions, heads, kv_heads, window, max(p + n for p, n in portions), 148) == (two < one)


@pytest.mark.parametrize("m,n,k,wide,library", [
    (777, 2048, 1536, 39.1, 111.5), (128, 512, 512, 26.0, 13.1), (2048, 8960, 1536, 390.0, 964.6), (64, 2048, 1536, 36.0, 29.8),
    (512, 512, 512, 17.0, 15.2), (1024, 1536, 8960, 220.0, 596.0), (32, 8960, 1536, 76.8, 33.5),
])
def test_float32_products_run_on_the_tensor_cores_where_that_is_faster(m, n, k, wide, library):
    assert wide_pays(m, n, k, 148) == (wide < library)


@pytest.mark.parametrize("rows,tile", [(12, 128), (75, 128), (112, 128), (131, 128), (169, 256), (188, 256), (394, 256), (562, 128), (750, 256)])
def test_routed_products_take_the_tile_that_is_not_slower(rows, tile):
    assert grouped_tile(16 * rows, 16) == tile


@pytest.mark.parametrize("experts,rows,single,pair", [  # us of a layer in tiles of 128 and of 256
    (8, 112, 76, 72), (8, 131, 76, 74), (8, 150, 84, 74), (8, 275, 106, 102), (8, 375, 111, 104), (8, 420, 119, 106),
    (16, 40, 313, 352), (16, 75, 320, 389), (16, 169, 422, 406), (16, 220, 428, 403), (16, 275, 565, 676), (16, 300, 662, 708), (16, 330, 678, 715),
    (16, 375, 182, 168), (16, 375, 723, 709), (16, 420, 862, 776), (16, 562, 1042, 1114), (16, 700, 1231, 1176),
    (64, 64, 298, 317), (64, 112, 344, 360), (64, 188, 436, 416), (64, 275, 596, 641), (64, 330, 668, 725), (64, 350, 686, 727), (64, 450, 883, 809),
    (64, 562, 1096, 1114), (64, 700, 1292, 1243),
])
def test_routed_products_take_the_tile_that_was_faster(experts, rows, single, pair):
    assert grouped_tile(experts * rows, experts) == (128 if single < pair else 256)


@pytest.fixture
def fake(monkeypatch):
    """A float32 kernel set on the CPU whose entries are only noted down; every float32 product pays."""
    entered = []
    monkeypatch.setattr(device, "wide_pays", lambda *args: True)
    monkeypatch.setattr(device, "function", lambda name: lambda *args: entered.append(name) or 0)
    ks = device.DeviceKernels.__new__(device.DeviceKernels)
    ks.dtype, ks.sm_count, ks.error_flag, ks.launches, ks.kernel_counts = torch.float32, 148, torch.zeros(1, dtype=torch.int32), 0, {}
    ks._stream = lambda: 0
    return ks, entered


def test_float32_products_that_the_library_refuses_or_spreads_stay_with_it(fake):
    """Operands that do not fit one another never reach the kernel, which takes its sizes from the weight alone."""
    ks, entered = fake
    x, w = torch.ones(200, 64), torch.ones(128, 64)
    ks.linear(x, w, torch.ones(128))
    assert entered and ks.kernel_counts == {"gemm_float32": 1}
    entered.clear()
    for wrong in (torch.ones(200, 56), torch.ones(200, 72), torch.ones(64), torch.ones(1, 200, 64)):
        with pytest.raises(RuntimeError):
            ks.linear(wrong, w)
    for bias in (torch.ones(127), torch.ones(129), torch.ones(200, 127)):
        with pytest.raises(RuntimeError):
            ks.linear(x, w, bias)
    with pytest.raises(RuntimeError):
        ks.linear(x, torch.ones(128, 64, 1))
    for bias in (torch.ones(1), torch.ones(1, 128), torch.ones(200, 128), torch.ones(200, 1)):
        assert torch.equal(ks.linear(x, w, bias), torch.full((200, 128), 65.0))
    grown = torch.ones(128, 64, requires_grad=True)
    ks.linear(x, grown).sum().backward()
    assert torch.equal(grown.grad, torch.full((128, 64), 200.0)) and not entered


def test_scratch_that_the_memory_does_not_hold_leaves_the_work_to_the_other_kernel(fake, monkeypatch):
    from distie_b200.kernels.interface import KvSlot, StepTensors

    ks, entered = fake
    sizes = {"distie_gemm_float32_scratch_floats": 1 << 50, "distie_attention_prefill_pairs_scratch_floats": 1 << 50}
    monkeypatch.setattr(device, "function", lambda name: lambda *args: entered.append(name) or sizes.get(name, 0))

    def full(*size, **kw):
        if size[0] == 1 << 50:
            raise torch.OutOfMemoryError("full")
        return torch.zeros(*size, **kw)

    monkeypatch.setattr(device.torch, "empty", full)
    assert torch.equal(ks.linear(torch.ones(200, 64), torch.ones(128, 64)), torch.full((200, 128), 64.0))
    assert entered == ["distie_gemm_float32_scratch_floats"]
    entered.clear()
    monkeypatch.setattr(device.DeviceKernels, "_in_pairs", lambda *args: True)
    ids = torch.zeros(2, dtype=torch.int32)
    step = StepTensors(token_ids=ids, positions=ids, token_seq=ids, seq_seat=ids, num_tokens=2, num_seqs=1, num_decode_tokens=0, max_kv_len=2)
    step.q_tiles, step.num_q_tiles = torch.tensor([[0, 2]], dtype=torch.int32), 1
    cache = torch.zeros(1, 1, 16, 64)
    q = torch.zeros(2, 64)
    assert ks._attention_tcgen05(q, q, step, KvSlot(cache, cache, ids[None], 16, 1), 1, 1, 64, 0, 0, 0.125)
    assert entered == ["distie_attention_prefill_pairs_scratch_floats", "distie_attention_prefill_tcgen05"]
    assert ks.kernel_counts == {"attention_prefill_tcgen05": 1} and ks.launches == 1
