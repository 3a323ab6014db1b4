"""The exponential gates under a running maximum over several chunks of a portion, against the plain recurrence in 64 bits.

The exponents are sums of the running maximum, at most the cap in size, with gates: each step rounds at cap * 2^-24, in
quadrature sqrt(tokens) of that, and a chunk's sum of gates once more as much; the bound is four times the first."""

from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import step_of

pytestmark = pytest.mark.gpu

CAP = 6.0


def exact(gates, bias, state):
    """gates [2, n, heads], state [heads] -> (keep, take, floor [3, n, heads], the maximum behind)"""
    i = CAP * torch.tanh((gates[0].double() + bias[0].double()) / CAP)
    f = torch.nn.functional.logsigmoid(CAP * torch.tanh((gates[1].double() + bias[1].double()) / CAP))
    m, rows = state.double(), []
    for t in range(i.shape[0]):
        new = torch.maximum(f[t] + m, i[t])
        rows.append(torch.stack([torch.exp(f[t] + m - new), torch.exp(i[t] - new), torch.exp(-new)]))
        m = new
    return torch.stack(rows, 1), m


# What the requests bring, step after step: portions at and off the edges of chunks of 8 to 64 tokens, alone and beside
# single tokens; heads that leave a block whole chunks, 63 tokens, and 8 with all of its shared memory.
STEPS = [
    [[64], [65], [129]],
    [[700, 1, 1], [1, 64, 129], [3, 1, 1]],
    [[1500, 300, 1, 2200], [1, 1, 1, 1], [40, 9, 1, 72]],
]


@pytest.mark.parametrize("steps", STEPS)
@pytest.mark.parametrize("heads,slices", [(5, 1), (5, 3), (65, 1), (512, 1)])
def test_gates_of_several_chunks(steps, heads, slices):
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(21)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    requests = len(steps[0])
    # head 0 hardly forgets and hardly takes (the maximum comes from far back), head 1 takes at every token
    bias = torch.stack([normal(heads), normal(heads) + 2])
    bias[:, 0], bias[:, 1] = torch.tensor([-20.0, 20.0]), torch.tensor([9.0, -9.0])
    state = normal(requests, heads)
    want_state, done = state.clone().double(), [0] * requests
    for lengths in steps:
        step = step_of(lengths, done, list(range(requests)))
        gates = normal(2, step.num_tokens, heads) * 3
        both = torch.cat([gates[0], gates[1]], -1)
        split = normal(slices, *both.shape)
        split[0] += both - split.sum(0)
        keep, take, floor = ks.exp_gate_scan(split[:, :, :heads], split[:, :, heads:], bias[0], bias[1], CAP, state, step)
        gates = split.double().sum(0).view(-1, 2, heads).transpose(0, 1)
        start = 0
        for row in sorted(range(requests), key=lambda i: (lengths[i] != 1, i)):
            end = start + lengths[row]
            want, want_state[row] = exact(gates[:, start:end], bias, want_state[row])
            got = torch.stack([keep, take, floor])[:, start:end].double()
            bound = (4 * (sum(s[row] for s in steps) ** 0.5) * CAP + 6 * slices) * 2**-24
            error = float(((got - want).abs() / want.abs().clamp_min(1e-30)).max())
            assert error <= bound, f"{lengths} request {row}: off by {error:.2e}, bound {bound:.2e}"
            start = end
        assert float((state.double() - want_state).abs().max()) <= 4 * 3000**0.5 * CAP * 2**-24
        done = [a + b for a, b in zip(done, lengths)]
