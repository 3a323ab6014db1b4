"""Linear recurrences of long portions (chunks on the tensor cores) against the token-by-token formulas in 64 bits.

The operands enter in three bfloat16 parts, which hold the 24 bits of a float32, so what is left is the rounding of
float32 sums and of a chunk's products of decays: at most 64 factors and 128 terms of 2^-24 each, in quadrature about
14 * 2^-24 = 8e-7 of the result; the bound is twice that.  The walk is held to the same bound."""

from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import step_of

pytestmark = pytest.mark.gpu

BOUND = 1.7e-6


def exact(rule, p, lengths, order, heads, groups, key_dim, value_dim, unit):
    double = {n: t.double() if t is not None else None for n, t in p.items()}
    wide = lambda x: x.reshape(-1, groups, key_dim).repeat_interleave(heads // groups, 1)  # noqa: E731
    q, k = wide(double["q"]), wide(double["k"])
    v = double["v"].reshape(q.shape[0], heads, -1)
    if unit:
        v = torch.cat([v, torch.ones_like(v[..., :1])], -1)
    softplus = torch.nn.functional.softplus
    if rule == "gated":
        g = double["decay"] if double["decay"] is not None else double["rate"].expand(q.shape[0], -1)
        factor = double["write"] if double["write"] is not None else torch.ones_like(g)
    elif rule == "ssd":
        factor = softplus(double["write"] + double["bias"])
        g = torch.exp(-double["rate"].exp() * factor)
    else:
        factor = torch.sigmoid(double["write"])
        g = torch.exp(-double["rate"].exp() * softplus(double["decay"] + double["bias"]))
        q = q / (q.square().sum(-1, keepdim=True) + 1e-6).sqrt() * key_dim**-0.5
        k = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    out = torch.empty(q.shape[0], heads, value_dim, dtype=torch.float64, device="cuda")
    states, start = double["state"].clone(), 0
    for row in order:
        S = states[row]
        for t in range(start, start + lengths[row]):
            S = S * g[t, :, None, None]
            held = torch.einsum("hvk,hk->hv", S, k[t]) if rule == "delta" else 0.0
            S = S + (factor[t, :, None] * (v[t] - held))[:, :, None] * k[t][:, None]
            out[t] = torch.einsum("hvk,hk->hv", S, q[t])
            if rule == "ssd":
                out[t] += double["skip"][:, None] * v[t]
        states[row] = S
        start += lengths[row]
    return out.reshape(q.shape[0], -1), states


# lengths, heads, groups, key size, value size: whole and ragged chunks, a token alone beside portions, sizes that fill no
# tile and no vector, the largest sizes taken, and one key size beyond them (the walk)
SIZES = [
    ([490], 4, 4, 128, 128),
    ([1, 257, 1, 193, 320], 4, 2, 64, 96),
    ([917], 2, 1, 50, 33),
    ([961], 2, 2, 17, 144),
    ([513, 64, 700], 3, 3, 128, 129),
    ([300], 2, 2, 160, 64),
]


@pytest.mark.parametrize("lengths,heads,groups,key_dim,value_dim", SIZES)
@pytest.mark.parametrize("rule,strong", [("delta", False), ("delta", True), ("ssd", False), ("ssd", True),
                                         ("gated", False), ("gated", True), ("constant", False)])
def test_chunks_of_a_recurrence(rule, strong, lengths, heads, groups, key_dim, value_dim):
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(7)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    total, constant = sum(lengths), rule == "constant"
    rule = "gated" if constant else rule
    unit = rule == "gated" and value_dim == 129
    p = {"q": normal(total, groups * key_dim), "k": normal(total, groups * key_dim) + 0.3,
         "v": normal(total, heads * (value_dim - unit)), "decay": normal(total, heads), "write": normal(total, heads),
         "rate": normal(heads) * 0.5, "bias": normal(heads) - 3, "skip": None,
         "state": normal(len(lengths), heads, value_dim, key_dim)}
    if rule == "delta" and strong:  # hardly anything is forgotten and all is corrected: the longest way through a chunk
        p["bias"], p["write"] = p["bias"] - 3, p["write"].abs() + 3
    if rule == "ssd":
        p["skip"] = normal(heads)
        p["bias"] += 6 if strong else 0  # strong: a token forgets nearly all that was before it
    elif rule == "gated" and not constant:
        p["decay"], p["write"] = torch.exp(-p["decay"] ** 2 * (9 if strong else 0.02)), torch.sigmoid(p["write"])
        if strong:
            p["decay"][normal(total, heads) > 2] = 0.0
    if constant:
        p["decay"] = p["write"] = None
        p["rate"] = torch.linspace(0.75, 0.996, heads, device="cuda")
    step = step_of(lengths, [3] * len(lengths), list(range(len(lengths))))
    order = sorted(range(len(lengths)), key=lambda i: (lengths[i] != 1, i))
    want, want_state = exact(rule, p, lengths, order, heads, groups, key_dim, value_dim, unit)
    state = p["state"].clone()
    got = ks.linear_recurrence(rule, p["q"].clone(), p["k"].clone(), p["v"], p["decay"], p["write"], state, step, heads, groups,
                               key_dim, value_dim, decay_rate=p["rate"], decay_bias=p["bias"] if rule != "gated" else None,
                               skip=p["skip"], unit_column=unit)
    assert ("recurrence_chunks" in ks.kernel_counts) == (key_dim <= 128)
    for name, a, b in (("read-out", got, want), ("state", state, want_state)):
        error = float((a.double() - b).norm() / b.norm())
        assert error <= BOUND, f"{rule} {name}: off by {error:.2e}"


def inputs(rule, lengths, heads, groups, key_dim, value_dim, seed=7):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    total = sum(lengths)
    p = {"q": normal(total, groups * key_dim), "k": normal(total, groups * key_dim) + 0.3, "v": normal(total, heads * value_dim),
         "decay": normal(total, heads), "write": normal(total, heads), "rate": normal(heads) * 0.5, "bias": normal(heads) - 3,
         "skip": normal(heads) if rule == "ssd" else None, "state": normal(len(lengths), heads, value_dim, key_dim)}
    if rule == "gated":
        p["decay"], p["write"] = torch.exp(-p["decay"] ** 2 * 0.02), torch.sigmoid(p["write"])
    return p


def run(ks, rule, p, lengths, heads, groups, key_dim, value_dim, state=None):
    state = p["state"].clone() if state is None else state
    got = ks.linear_recurrence(rule, p["q"], p["k"], p["v"], p["decay"], p["write"], state,
                               step_of(lengths, [3] * len(lengths), list(range(len(lengths)))), heads, groups, key_dim, value_dim,
                               decay_rate=p["rate"], decay_bias=p["bias"] if rule != "gated" else None, skip=p["skip"])
    ks.check_errors()
    assert "recurrence_chunks" in ks.kernel_counts and "linear_recurrence" not in ks.kernel_counts
    return got, state


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "decay", "write", "state"])
@pytest.mark.parametrize("rule", ["delta", "ssd", "gated"])
def test_a_number_that_is_not_finite_spoils_its_token_and_those_behind_it(rule, where, bad):
    """As in the walk: nothing before the token, no other request, no column of a state that does not meet it."""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    lengths, heads, groups, key_dim, value_dim = [300, 257, 200], 4, 2, 64, 48
    p = inputs(rule, lengths, heads, groups, key_dim, value_dim)
    if where == "state":
        p["state"][0, 1, 5, 7] = bad
    else:
        p[where][100, 1], p[where][300 + 256, 0] = bad, bad  # inside a chunk; the last token of a request
    want, want_state = exact(rule, p, lengths, range(3), heads, groups, key_dim, value_dim, False)
    got, state = run(ks, rule, p, lengths, heads, groups, key_dim, value_dim)
    for name, a, b in (("read-out", got, want), ("state", state, want_state)):
        fine = torch.isfinite(b)
        assert fine.any() and torch.equal(torch.isfinite(a), fine), f"{name}: other numbers are spoiled"
        error = float((a.double() - b)[fine].norm() / b[fine].norm())
        assert error <= BOUND, f"{name}: off by {error:.2e}"


@pytest.mark.parametrize("rule", ["delta", "ssd", "gated"])
def test_portions_beyond_the_scratch_run_in_groups_of_tiles(rule, monkeypatch):
    """Groups that end inside a request and between two: the same arithmetic, so the same numbers."""
    from distie_b200.kernels import device, make_kernels

    lengths, heads, groups, key_dim, value_dim = [640, 300, 385, 140], 4, 2, 64, 48
    p = inputs(rule, lengths, heads, groups, key_dim, value_dim)  # 5 + 3 + 4 + 2 tiles
    whole, whole_state = run(make_kernels(torch.bfloat16, "cuda:0"), rule, p, lengths, heads, groups, key_dim, value_dim)
    of_tile = device.function("distie_recurrence_chunks_scratch_floats")(device._RULES[rule], 1, heads, key_dim, value_dim)
    for tiles in (1, 3, 13):
        monkeypatch.setattr(device, "_CHUNK_BYTES", 4 * of_tile * tiles + 3)
        ks = make_kernels(torch.bfloat16, "cuda:0")
        got, state = run(ks, rule, p, lengths, heads, groups, key_dim, value_dim)
        assert ks.kernel_counts["recurrence_chunks"] == -(-14 // tiles)
        assert torch.equal(got, whole) and torch.equal(state, whole_state)


@pytest.mark.parametrize("rule", ["delta", "ssd", "gated"])
@pytest.mark.parametrize("slices,offset,extra", [(3, 0, 0), (1, 1, 3), (3, 1, 0)])
def test_slices_and_addresses_that_no_vector_fits(rule, slices, offset, extra):
    """Decay and write as slices of one projection; rows of q, k and v and the state a float off 16 bytes, rows of any stride.
    Adding up three slices rounds twice more, in a gate that a chunk multiplies up to 64 times: twice the bound."""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    lengths, heads, groups, key_dim, value_dim = [300, 257, 200], 4, 2, 64, 48
    p = inputs(rule, lengths, heads, groups, key_dim, value_dim)
    total, columns = sum(lengths), 2 * groups * key_dim + heads * value_dim
    rows = torch.full((total, offset + columns + extra), float("nan"), device="cuda")[:, offset : offset + columns]
    rows.copy_(torch.cat([p["q"], p["k"], p["v"]], -1))
    p["q"], p["k"], p["v"] = rows.split([groups * key_dim, groups * key_dim, heads * value_dim], -1)
    both = torch.cat([p["decay"], p["write"]], -1)
    gates = torch.empty(slices, total, 2 * heads + 1, device="cuda")[:, :, : 2 * heads]
    for s in range(1, slices):
        gates[s] = both * (0.2 * s)
    gates[0] = both - gates[1:].sum(0)
    if rule == "gated":  # (a decay stays what it was: at most 1)
        gates[0, :, :heads] = torch.minimum(gates[0, :, :heads], 1 - gates[1:, :, :heads].sum(0))
    summed = gates.double().sum(0)
    held = torch.empty(p["state"].numel() + offset, device="cuda")[offset:].view_as(p["state"]).copy_(p["state"])
    want, want_state = exact(rule, p | {"decay": summed[:, :heads], "write": summed[:, heads:]}, lengths, range(3), heads, groups,
                             key_dim, value_dim, False)
    p["decay"], p["write"] = gates[:, :, :heads], gates[:, :, heads:]
    got, state = run(ks, rule, p, lengths, heads, groups, key_dim, value_dim, held)
    for name, a, b in (("read-out", got, want), ("state", state, want_state)):
        error = float((a.double() - b).norm() / b.norm())
        assert error <= (2 if slices > 1 else 1) * BOUND, f"{name}: off by {error:.2e}"


@pytest.mark.parametrize("lengths,heads,key_dim,value_dim", [([917], 2, 128, 128), ([513, 64, 700], 3, 64, 143), ([400, 333], 4, 128, 40)])
@pytest.mark.parametrize("offset,extra", [(0, 0), (1, 2)])
def test_a_stabilised_memory_in_one_go(lengths, heads, key_dim, value_dim, offset, extra):
    """The projection as it is: q scaled on the way in, read-outs divided on the way out, by the normaliser in some rows
    and by the floor in others.  A divisor is at least 0.3 of the normaliser's size, so its error counts up to 1 / 0.3 times."""
    from distie_b200.kernels import make_kernels

    ks = make_kernels(torch.bfloat16, "cuda:0")
    generator = torch.Generator(device="cuda").manual_seed(17)
    normal = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    total, columns, scale = sum(lengths), heads * (2 * key_dim + value_dim), key_dim**-0.5
    rows = torch.full((total, offset + columns + extra), float("nan"), device="cuda")[:, offset : offset + columns]
    rows.copy_(normal(total, columns))
    keep, take = torch.exp(-normal(total, heads) ** 2 * 0.02), torch.sigmoid(normal(total, heads))
    state = normal(len(lengths), heads, value_dim + 1, key_dim)
    q, k, v = rows.split([heads * key_dim, heads * key_dim, heads * value_dim], -1)
    read, want_state = exact("gated", {"q": q.double() * scale, "k": k, "v": v, "decay": keep, "write": take, "state": state}, lengths,
                             range(len(lengths)), heads, heads, key_dim, value_dim + 1, True)
    read = read.view(total, heads, value_dim + 1)
    size = read[:, :, value_dim].abs()
    floor = (size * torch.where(normal(total, heads) > 0, 1.5, 0.5)).clamp_min(0.3 * float(size.square().mean().sqrt())).float()
    assert 0.3 < float((floor > size).float().mean()) < 0.8
    want = (read[:, :, :value_dim] / (torch.maximum(size, floor.double()) + 1e-6)[:, :, None]).reshape(total, -1)
    step = step_of(lengths, [3] * len(lengths), list(range(len(lengths))))
    got = ks.stabilized_memory(rows, scale, keep, take, floor, state, step, heads, key_dim, value_dim)
    ks.check_errors()
    assert "recurrence_chunks" in ks.kernel_counts and not {"linear_recurrence", "stabilized_readout"} & set(ks.kernel_counts)
    for name, a, b, bound in (("read-out", got, want, (1 + 1 / 0.3) * BOUND), ("state", state, want_state, BOUND)):
        error = float((a.double() - b).norm() / b.norm())
        assert error <= bound, f"{name}: off by {error:.2e}"
