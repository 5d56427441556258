"""Float32 attention of prompts on the tensor cores (three bfloat16 parts a number) against 64 bits, and what numbers it does not
take fall back to."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
D = 64


def ops():
    from gpullama3.java_b200.kernels import ops as o
    return o


def case(q_lens, behind, H, G, seed, std=1.0):
    g = torch.Generator("cuda").manual_seed(seed)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n, kv = len(q_lens), [b + q for b, q in zip(behind, q_lens)]
    W = max(-(-k // 64) for k in kv) + 1                     # (a column that no sequence uses yet)
    table = torch.randperm(n * W + 3, generator=torch.Generator().manual_seed(seed))[:n * W].to(torch.int32).view(n, W).cuda()
    k_pool, v_pool = randn(n * W + 3, G, 64, D) * std, randn(n * W + 3, G, D, 64)
    qkv = randn(sum(q_lens), (H + 2 * G) * D) * std
    cu = torch.tensor([0] + torch.tensor(q_lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    return qkv, cu, torch.tensor(kv, dtype=torch.int32, device="cuda"), table, k_pool, v_pool


def both(c, q_lens, H, G):
    o = ops()
    qkv, rest = c[0], c[1:]
    outs = [torch.full((qkv.shape[0], H * D), 7.0, device="cuda") for _ in range(2)]
    args = (*rest, len(q_lens), max(q_lens), H, G, D)
    assert o.attention_prefill_f32_tc(qkv, qkv.shape[1], outs[0], *args)
    assert o.attention_prefill_f32(qkv, qkv.shape[1], outs[1], *args, tile=32, n_spans=1)
    assert o.attention_prefill_f32_tc_status() == 0
    return outs


def exact(c, q_lens, behind, H, G):
    qkv, cu, kv_lens, table, k_pool, v_pool = c
    out = torch.empty(qkv.shape[0], H, D, dtype=torch.float64, device="cuda")
    n, W = table.shape
    k = k_pool[table.long()].permute(0, 2, 1, 3, 4).reshape(n, G, W * 64, D).double()
    v = v_pool[table.long()].permute(0, 2, 3, 1, 4).reshape(n, G, D, W * 64).double()
    for s in range(n):
        rows, kv = slice(int(cu[s]), int(cu[s + 1])), behind[s] + q_lens[s]
        hidden = torch.arange(kv, device="cuda")[None] > torch.arange(behind[s], kv, device="cuda")[:, None]
        for h in range(H):
            scores = qkv[rows, h * D:(h + 1) * D].double() @ k[s, h // (H // G), :kv].T / 8
            out[rows, h] = scores.masked_fill(hidden, -math.inf).softmax(-1) @ v[s, h // (H // G), :, :kv].T
    return out.reshape(-1, H * D)


@pytest.mark.parametrize("q_lens, behind, H, G", [([1], [0], 2, 1), ([64], [0], 4, 2), ([127, 65], [1, 63], 4, 2), ([128], [64], 8, 2),
                                                  ([129, 1, 300], [700, 64, 5], 6, 1), ([2048], [0], 32, 8), ([700] * 3, [0, 1, 100], 16, 4)])
@pytest.mark.parametrize("std", [1.0, 2.5], ids=["mild", "peaked"])
def test_against_64_bits(q_lens, behind, H, G, std):
    """Rows of one to 128 in a tile, pages begun and ended anywhere, CTAs with several tiles.  The probabilities' own rounding and the
    scores' (2^-24 of scores of a few std^2) are common to both kernels; the products and sums here must not add to what the
    multiply-add kernel leaves, up to the spread of that figure over inputs of few rows."""
    c = case(q_lens, behind, H, G, sum(q_lens) + H, std)
    want = exact(c, q_lens, behind, H, G)
    got, tiles = both(c, q_lens, H, G)
    err = [float((x.double() - want).norm() / want.norm()) for x in (got, tiles)]
    assert err[0] <= 1.25 * err[1], err


@pytest.mark.parametrize("what", ["inf value", "nan key", "huge query", "huge value", "tiny values"])
def test_numbers_without_such_parts(what):
    """Numbers that are not finite, or too large for sums of parts, go to the multiply-add kernel: its bits.  Values far below 1 keep
    float32's relative precision."""
    q_lens, behind, H, G = [150, 70], [20, 0], 4, 2
    c = case(q_lens, behind, H, G, 5)
    qkv, cu, kv_lens, table, k_pool, v_pool = c
    page = int(table[0, 1])
    if what == "inf value":
        v_pool[page, 0, 3, 5] = math.inf
    elif what == "nan key":
        k_pool[page, 1, 7, 5] = math.nan
    elif what == "huge query":
        qkv[5, 70] = 1e25
    elif what == "huge value":
        v_pool[page, 1, 3, 5] = 3e36
    else:
        v_pool *= 1e-36
    got, tiles = both(c, q_lens, H, G)
    if what == "tiny values":
        want = exact(c, q_lens, behind, H, G)
        err = [float((x.double() - want).norm() / want.norm()) for x in (got, tiles)]
        assert err[0] <= 1.25 * err[1], err
    else:
        assert torch.equal(got.isnan(), tiles.isnan()) and torch.equal(got.nan_to_num(), tiles.nan_to_num())


@pytest.mark.parametrize("keys", [64, 2048])
@pytest.mark.parametrize("value", [1e30, 2.0 ** 72, 2.0 ** 71.9, -2.0 ** 71.9, 1e20], ids=["1e30", "at the bound", "below it", "negative", "1e20"])
def test_large_values_of_equal_weight(value, keys):
    """Scores of 0, so that a row's unnormalised sum grows with its keys: finite at every length, and from the bound on (2^72) the
    multiply-add kernel's bits.  Below it every row is the mean of equal values: each of the twelve products that are added up for half a page cuts off at most
    2^-23 of the sum, all to the same side where the values are equal."""
    q_lens, behind, H, G = [128], [keys - 128], 4, 2
    if keys < 128:
        q_lens, behind = [keys], [0]
    c = case(q_lens, behind, H, G, 7)
    c[0].zero_()
    c[5].fill_(value)
    got, tiles = both(c, q_lens, H, G)
    assert bool(got.isfinite().all())
    if value >= 2.0 ** 72:
        assert torch.equal(got, tiles)
    else:
        torch.testing.assert_close(got, torch.full_like(got, value), rtol=12 * 2.0 ** -23, atol=0.0)


def test_stale_pages_are_not_read():
    """What lies behind a sequence's end in its last page, and pages it does not have, may hold anything."""
    q_lens, behind, H, G = [100], [30], 4, 2
    c = case(q_lens, behind, H, G, 9)
    qkv, cu, kv_lens, table, k_pool, v_pool = c
    want = exact(c, q_lens, behind, H, G)
    last = int(table[0, 2])
    k_pool[last, :, 2:], v_pool[last, :, :, 2:] = math.nan, math.inf
    table[0, 3] = 2 ** 30
    got, _ = both((qkv, cu, kv_lens, table[:, :3].contiguous(), k_pool, v_pool), q_lens, H, G)
    assert float((got.double() - want).norm() / want.norm()) < 1e-6


def test_declines_what_it_does_not_take():
    o = ops()
    c = case([64], [0], 3, 1, 1)
    out = torch.empty(64, 3 * D, device="cuda")
    assert not o.attention_prefill_f32_tc(c[0], c[0].shape[1], out, *c[1:], 1, 64, 3, 1, D)
