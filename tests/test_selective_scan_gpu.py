"""Which B and C the selective scan of a portion takes: views of the slices of one projection, wherever they lie in it."""

from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import step_of

pytestmark = pytest.mark.gpu

CHANNELS, STATES, RANK = 96, 16, 8


def _run(lengths, place):
    """The scan with ``place(numbers [S, T, 2 states]) -> (B, C)``; (output, state)"""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(2)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    step = step_of(lengths, [3] * len(lengths), list(range(len(lengths))))
    tokens = step.num_tokens
    x, dt, gate = normal(tokens, CHANNELS), normal(1, tokens, CHANNELS) - 2, normal(tokens, CHANNELS)
    numbers, state = normal(3, tokens, 2 * STATES), normal(len(lengths), STATES, CHANNELS)
    rates, skip, bias = -torch.rand(STATES, CHANNELS, generator=generator, device="cuda") - 0.1, normal(CHANNELS), normal(CHANNELS)
    out = torch.empty(tokens, CHANNELS, dtype=torch.bfloat16, device="cuda")
    B, C = place(numbers)
    ks.selective_scan(x, dt, B, C, gate, rates, skip, bias, state, step, out)
    ks.check_errors()
    return out, state


def _in(numbers, columns, b_at, c_at):
    wide = torch.full((*numbers.shape[:2], columns), float("nan"), device="cuda")
    wide[:, :, b_at : b_at + STATES], wide[:, :, c_at : c_at + STATES] = numbers[:, :, :STATES], numbers[:, :, STATES:]
    return wide[:, :, b_at : b_at + STATES], wide[:, :, c_at : c_at + STATES]


@pytest.mark.parametrize("lengths", [[300], [1, 70, 1, 260], [4]])
def test_b_and_c_anywhere_in_a_projection(lengths):
    neighbours = _run(lengths, lambda numbers: _in(numbers, RANK + 2 * STATES, RANK, RANK + STATES))
    for columns, b_at, c_at in ((2 * STATES, STATES, 0), (3 * STATES + 4, 0, 2 * STATES)):
        out, state = _run(lengths, lambda numbers: _in(numbers, columns, b_at, c_at))
        # (the same numbers; slices are added in the same order, so the float32 state is the same to its last bits)
        assert float((state - neighbours[1]).abs().max()) <= 1e-5
        assert float((out.float() - neighbours[0].float()).norm() / neighbours[0].float().norm()) <= 2**-9


def test_b_and_c_of_different_layouts_are_refused():
    from distie_b200.kernels.library import KernelError

    with pytest.raises(KernelError):
        _run([300], lambda numbers: (_in(numbers, RANK + 2 * STATES, 0, STATES)[0], numbers[:, :, STATES:].contiguous()))
