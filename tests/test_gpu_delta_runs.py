"""The gated delta rule in runs of tokens, against its recurrence in 64 bits and against the kernel that takes a token at a
time: run ends, sequences shorter than a run beside long ones, key heads shared by heads, decays that underflow within a
run, value sizes of several tiles, numbers that are not finite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def recurrence(qkv, beta, decay, dt_bias, a_log, states, lengths, H, G, dk, dv, per_head):
    x, outs, finals, at = qkv.double(), [], [], 0
    for S, n in zip(states, lengths):
        rows = slice(at, at + n)
        at += n
        q, k = (x[rows, i * G * dk:(i + 1) * G * dk].view(n, G, dk).repeat_interleave(H // G, 1) for i in (0, 1))
        v = x[rows, 2 * G * dk:].view(n, H, dv)
        unit = lambda y: y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)
        q, k, b = unit(q) * dk ** -0.5, unit(k), torch.sigmoid(beta[rows, :H].double())
        step = torch.nn.functional.softplus(decay[rows].double() + dt_bias.double())
        step = step[..., None].expand(n, H, dk) if per_head else step.view(n, H, dk)
        g = torch.exp(-torch.exp(a_log.double())[:, None] * step)
        S = S.double().clone()
        for t in range(n):
            S = S * g[t, :, :, None]
            u = b[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            outs.append(torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1))
        finals.append(S)
    return torch.stack(outs), torch.stack(finals)


def problem(lengths, H, G, dv, dtype, per_head, strong):
    gen = torch.Generator("cuda").manual_seed(sum(lengths) + H + dv)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    T, n, dk = sum(lengths), len(lengths), 64
    nd = H if per_head else H * dk
    return dict(qkv=rand(T, 2 * G * dk + H * dv).to(dtype), beta=rand(T, H + 3).to(dtype), decay=(rand(T, nd) * (3 if strong else 1)).to(dtype),
                dt_bias=rand(nd), a_log=rand(H) * 0.5 + (2 if strong else -1), state=rand(n, H * dk * dv + 32),
                slots=torch.randperm(n, generator=gen, device="cuda").to(torch.int32),
                cu=torch.tensor([0] + lengths).cumsum(0).to(torch.int32).cuda())


def scan(p, lengths, H, G, dv, per_head, longest):
    from gpullama3.java_b200.kernels import ops

    state, out = p["state"].clone(), torch.full((sum(lengths), H * dv), 9.0, device="cuda")
    asked = []

    def alloc(shape, dtype):
        asked.append(shape)
        return torch.empty(shape, dtype=dtype, device="cuda")

    ops.delta_rule_scan(p["qkv"], p["beta"], p["decay"], p["dt_bias"], p["a_log"], state, p["slots"], p["cu"], out, H, G, 64, dv, 64 ** -0.5,
                        1e-6, alloc=alloc, decay_per_head=per_head, longest=longest)
    return out, state, len(asked)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("lengths, H, G, dv, per_head, strong", [
    ([96], 2, 1, 16, False, False), ([97], 4, 4, 32, False, False), ([33, 1, 64, 200], 4, 2, 64, False, False), ([100, 31, 5, 127], 4, 4, 48, True, False),
    ([300], 4, 4, 128, False, True), ([31, 161], 3, 1, 80, True, True)])
def test_runs_of_tokens_against_the_recurrence(lengths, H, G, dv, per_head, strong, dtype):
    """A result is a few hundred 32-bit operations away from its inputs (a sum of 64 channels, 32 tokens of a run, one addition per
    run, the decays' functions), each of 2^-24 of terms no larger than the largest: 2^-14 of the largest is never reached, and the norm of all errors
    stays below 2^-20 of the results' (they add up like random steps)."""
    p = problem(lengths, H, G, dv, dtype, per_head, strong)
    live = H * 64 * dv
    want, states = recurrence(p["qkv"], p["beta"], p["decay"], p["dt_bias"], p["a_log"], [p["state"][s, :live].view(H, 64, dv) for s in p["slots"]],
                              lengths, H, G, 64, dv, per_head)
    out, state, allocations = scan(p, lengths, H, G, dv, per_head, max(lengths))
    assert allocations == 2                             # (the second: it went in runs)
    got = torch.stack([state[s, :live].view(H, 64, dv) for s in p["slots"]])
    for g, w in ((out, want), (got, states)):
        assert float((g.double() - w).norm() / w.norm()) < 2.0 ** -20
        assert float((g.double() - w).abs().max() / w.abs().max()) < 2.0 ** -14
    assert torch.equal(state[:, live:], p["state"][:, live:])
    one_by_one, state1, allocations = scan(p, lengths, H, G, dv, per_head, 1)
    assert allocations == 1
    assert float((one_by_one - out).norm() / out.norm()) < 2.0 ** -20


@pytest.mark.parametrize("what", ["q", "k", "v", "decay", "beta"])
def test_numbers_that_are_not_finite_reach_later_tokens_only(what):
    lengths, H, G, dv = [100, 96], 2, 2, 32
    p = problem(lengths, H, G, dv, torch.float32, False, False)
    clean, clean_state, _ = scan(p, lengths, H, G, dv, False, 100)
    target = {"q": (p["qkv"], 5), "k": (p["qkv"], 2 * 64 + 5), "v": (p["qkv"], 4 * 64 + 5), "decay": (p["decay"], 5), "beta": (p["beta"], 0)}[what]
    target[0][50, target[1]] = math.nan
    runs, state, _ = scan(p, lengths, H, G, dv, False, 100)
    one_by_one, state1, _ = scan(p, lengths, H, G, dv, False, 1)
    assert torch.equal(torch.isnan(runs), torch.isnan(one_by_one)) and torch.equal(torch.isnan(state), torch.isnan(state1))
    assert bool(torch.isnan(runs).any())
    assert torch.equal(runs[:50], clean[:50]) and torch.equal(runs[100:], clean[100:])


@pytest.mark.parametrize("per_head", [False, True], ids=["per channel", "per head"])
@pytest.mark.parametrize("kind", ["independent", "activated", "one sign", "weak decay", "dependent keys", "strong decay"])
def test_runs_are_no_further_from_64_bits_than_the_token_chain(kind, per_head):
    """The norm of all errors against the recurrence in 64 bits, over 500,000 results: what a token at a time leaves, and what runs leave.
    The states' errors are 65,000 numbers that mostly stem from the same roundings on both sides (unit rows, decays, the state's own):
    their norms differ by chance by up to one in a hundred, and a run's 32 writes to a state, of alternating signs where keys have one sign, are
    added up before they join it (a fiftieth more there): a twentieth is allowed.  Queries and keys of one sign make B U and
    (G q) S large and of opposite signs; keys that nearly depend on each other, written with full strength, make the triangular system stiff."""
    lengths, H, dv = [500], 16, 64
    p = problem(lengths, H, H, dv, torch.float32, per_head, kind == "strong decay")
    heads = H * 64
    qkv = p["qkv"]
    if kind == "activated":
        p["qkv"] = torch.nn.functional.silu(qkv)
    elif kind == "one sign":
        qkv[:, :2 * heads] = qkv[:, :2 * heads].abs() + 0.2
    elif kind == "weak decay":
        p["decay"] -= 6
        p["beta"] += 3
    elif kind == "dependent keys":
        qkv[:, heads:2 * heads] = qkv[:1, heads:2 * heads] + 0.3 * qkv[:, heads:2 * heads]
        p["decay"] -= 4
        p["beta"] += 4
    live = H * 64 * dv
    want, states = recurrence(p["qkv"], p["beta"], p["decay"], p["dt_bias"], p["a_log"], [p["state"][s, :live].view(H, 64, dv) for s in p["slots"]],
                              lengths, H, H, 64, dv, per_head)
    errors = []
    for longest, allocations in ((500, 2), (1, 1)):
        out, state, asked = scan(p, lengths, H, H, dv, per_head, longest)
        assert asked == allocations
        got = torch.stack([state[s, :live].view(H, 64, dv) for s in p["slots"]])
        errors.append([float((g.double() - w).norm()) for g, w in ((out, want), (got, states))])
    (runs, runs_state), (chain, chain_state) = errors
    assert runs <= chain and runs_state <= 1.05 * chain_state
