"""Decode-step forms: a delta-rule token with its output norm in one launch, attention groups that share a key/value head, and spans of
unequal sequences."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def ops():
    from gpullama3.java_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("H, G, T, per_head, activation", [(32, 32, 8, False, "sigmoid"), (4, 2, 1, True, "silu"), (3, 1, 70, False, "silu"),
                                                           (2, 2, 3, True, "sigmoid")])
def test_delta_rule_token_in_one_launch(dtype, H, G, T, per_head, activation):
    """Against the same token by the scan and the norm's kernel: the states to 32-bit rounding of sums of 64 (2^-24 of the terms' sum,
    a few times), the results to that and one rounding to the storage type."""
    o = ops()
    g = torch.Generator("cuda").manual_seed(H * T)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    d, channels = 64, (2 * G + H) * 64
    wide = randn(T, channels + 16 + 2 * H * 64 + 16).to(dtype)
    qkv, beta, decay, gate = wide[:, :channels].contiguous(), wide[:, channels:channels + H], wide[:, channels + 16:], wide[:, channels + 16 + H * d:]
    dt_bias, a_log, w = randn(H if per_head else H * d), randn(H) * 0.5 - 1, 1 + 0.1 * randn(d)
    slots = torch.randperm(T + 2, generator=torch.Generator().manual_seed(T))[:T].to(torch.int32).cuda()
    state0 = randn(T + 2, H * d * d + 24)
    cu = torch.arange(T + 1, dtype=torch.int32, device="cuda")
    want_state, raw, want = state0.clone(), torch.empty(T, H * d, device="cuda"), torch.empty(T, H * d, dtype=dtype, device="cuda")
    o.delta_rule_scan(qkv, beta, decay, dt_bias, a_log, want_state, slots, cu, raw, H, G, d, d, 0.125, 1e-6, decay_per_head=per_head)
    o.gated_rmsnorm(raw, w, gate, want, H, d, 1e-5, activation)
    got_state, got = state0.clone(), torch.empty_like(want)
    assert o.delta_rule_step(qkv, beta, decay, dt_bias, a_log, got_state, slots, w, gate, got, H, G, d, d, 0.125, 1e-6, 1e-5, per_head, activation)
    torch.testing.assert_close(got_state, want_state, rtol=1e-5, atol=2e-6)
    tol = dict(rtol=2.0 ** -7, atol=1e-5) if dtype == torch.bfloat16 else dict(rtol=3e-5, atol=3e-6)
    torch.testing.assert_close(got, want, **tol)
    assert not o.delta_rule_step(qkv, beta, decay, dt_bias, a_log, got_state, slots, w, gate, got, H, G, 32, d, 0.125, 1e-6, 1e-5, per_head, activation)


def paged(lens, G, D, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    W = -(-max(lens) // 64)
    n = len(lens) * W
    table = torch.randperm(n + 1, generator=torch.Generator().manual_seed(seed))[:n].to(torch.int32).view(len(lens), W).cuda()
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    return torch.tensor(lens, dtype=torch.int32, device="cuda"), table, randn(n + 1, G, 64, D), randn(n + 1, G, D, 64), randn


@pytest.mark.parametrize("D, groups, splits", [(128, 2, 4), (96, 3, 1), (64, 2, 2)])
@pytest.mark.parametrize("terms", [False, True])
def test_groups_that_share_a_kv_head(D, groups, splits, terms):
    """All groups in one launch: the bits of a launch per group."""
    o = ops()
    lens, H = [700, 33, 1, 260], 16 * groups
    kv_lens, table, k, v, randn = paged(lens, 1, D, D + groups)
    q, gate, sinks = randn(len(lens), H * D), randn(len(lens), H), torch.linspace(-1, 1, H, device="cuda")
    got = torch.empty(len(lens), H * D, dtype=torch.bfloat16, device="cuda")
    extra = lambda s: dict(sinks=sinks[s].contiguous(), gate=gate[:, s]) if terms else {}
    o.attention_decode(q, H * D, got, kv_lens, table, k, v, H, groups, D, 0, splits, pool_heads=1, **extra(slice(0, H)))
    for i in range(groups):
        s = slice(16 * i, 16 * i + 16)
        part = torch.empty(len(lens), 16 * D, dtype=torch.bfloat16, device="cuda")
        o.attention_decode(q[:, 16 * i * D:], H * D, part, kv_lens, table, k, v, 16, 1, D, 0, splits, **extra(s))
        assert torch.equal(got[:, 16 * i * D:16 * (i + 1) * D], part)


@pytest.mark.parametrize("lens, splits", [([218, 1463, 942, 1029, 117, 1633, 2026, 687], 4), ([1] * 40 + [3000], 2), ([64 * i + 1 for i in range(64)], 4),
                                          ([33, 4000], 64), ([5] * 3, 8), ([777] * 65, 2)])
@pytest.mark.parametrize("window", [0, 500])
def test_spans_of_unequal_sequences(lens, splits, window):
    o = ops()
    H, G, D = 8, 2, 64
    kv_lens, table, k, v, randn = paged(lens, G, D, len(lens) + splits)
    q, out = randn(len(lens), H * D), torch.empty(len(lens), H * D, dtype=torch.bfloat16, device="cuda")
    o.attention_decode(q, H * D, out, kv_lens, table, k, v, H, G, D, window, splits)
    for i, n in enumerate(lens):
        lo = max(0, n - window) if window else 0
        ks = k[table[i].long()].permute(1, 0, 2, 3).reshape(G, -1, D)[:, lo:n].double()
        vs = v[table[i].long()].permute(1, 0, 3, 2).reshape(G, -1, D)[:, lo:n].double()
        s = torch.einsum("hd,hnd->hn", q[i].view(H, D).double(), ks.repeat_interleave(H // G, 0)) / math.sqrt(D)
        want = torch.einsum("hn,hnd->hd", s.softmax(-1), vs.repeat_interleave(H // G, 0)).reshape(-1)
        # (probabilities and results rounded to bfloat16)
        torch.testing.assert_close(out[i].double(), want, rtol=2.0 ** -7, atol=2.0 ** -7)
