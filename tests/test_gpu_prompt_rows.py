"""Prompt forms of the kernels between a mixer's products: stream connections through a ring of stages, head rows in tiles without
angles, output norms of several rows a warp, convolutions over runs, and windows in the attention over pairs of tiles."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def ops():
    from gpullama3.java_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("streams, width, T", [(3, 2048, 592), (3, 2048, 2048), (1, 64, 700), (2, 4096, 601), (4, 2052, 777), (8, 300, 600), (5, 260, 595)])
@pytest.mark.parametrize("reads", [True, False])
def test_streams_step_through_a_ring(streams, width, T, reads):
    """The same bits as the kernel of fewer tokens, which takes the rows in pieces."""
    o = ops()
    g = torch.Generator("cuda").manual_seed(T + width)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, y, mix, write, read, w = randn(T, streams, width), randn(T, width), randn(streams, streams), randn(streams), randn(streams), randn(width)

    def run(piece):
        xs, ys, out = x.clone(), y.clone(), torch.zeros(T, width, dtype=torch.bfloat16, device="cuda")
        for at in range(0, T, piece):
            part = slice(at, min(T, at + piece))
            o.streams_step(xs[part], mix, write, ys[part], *((read, w, out[part], 1e-6) if reads else ()))
        return xs, ys, out
    whole, pieces = run(T), run(300)
    for a, b in zip(whole, pieces):
        assert torch.equal(a, b)
    assert not whole[1].any()
    assert o.streams_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("H, G, d, D, T", [(32, 8, 64, 64, 300), (3, 1, 40, 64, 257), (2, 2, 128, 128, 2048), (5, 5, 248, 256, 256)])
def test_head_rows_of_many_tokens_without_angles(H, G, d, D, T, dtype):
    """Queries with bias, norm and factor to a buffer widened with zeros, keys and values into their pages."""
    o = ops()
    g = torch.Generator("cuda").manual_seed(T + d)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    raw = randn(T, (H + 2 * G) * d).to(dtype)
    bias, weight = randn((H + 2 * G) * d), randn(2 * d)
    W = -(-(T + 5) // 64)
    table = torch.randperm(W + 2, generator=torch.Generator().manual_seed(T))[:W].to(torch.int32).view(1, W).cuda()
    positions = torch.arange(5, T + 5, dtype=torch.int32, device="cuda")
    k_pool, v_pool = (torch.full(s, 3.0, dtype=dtype, device="cuda") for s in ((W + 2, G, 64, D), (W + 2, G, D, 64)))
    seg = o.head_row_segment
    segments = o.head_row_segments(seg(0, H, d, 0, D, 0, True, 0, 0.25), seg(H * d, G, d, 0, D, H * d, True, d, target=o.TO_CACHE_KEYS),
                                   seg((H + G) * d, G, d, 0, D, (H + G) * d, False, -1, target=o.TO_CACHE_VALUES))
    dst = torch.full((T, H * D), 5.0, dtype=dtype, device="cuda")
    o.head_rows(raw, dst, segments, 1e-6, bias, weight, cache=(positions, torch.zeros_like(positions), table, k_pool, v_pool))
    z = raw.double() + bias.double()
    unit = lambda r: r / torch.sqrt((r * r).mean(-1, keepdim=True) + 1e-6)
    pad = lambda r: torch.nn.functional.pad(r, (0, D - d))
    q = pad(unit(z[:, :H * d].view(T, H, d)) * weight[:d].double() * 0.25).reshape(T, -1)
    k = pad(unit(z[:, H * d:(H + G) * d].view(T, G, d)) * weight[d:].double())
    v = pad(z[:, (H + G) * d:].view(T, G, d))
    page, at = table[0].long()[positions.long() // 64], positions.long() % 64
    tol = dict(rtol=2.0 ** -8, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=2e-6, atol=2e-6)
    torch.testing.assert_close(dst.double(), q, **tol)
    torch.testing.assert_close(k_pool[page, :, at].double(), k, **tol)
    torch.testing.assert_close(v_pool[page, :, :, at].double(), v, **tol)
    untouched = torch.ones(W + 2, 64, dtype=torch.bool, device="cuda")
    untouched[page, at] = False
    assert bool((k_pool.permute(0, 2, 1, 3)[untouched] == 3.0).all()) and bool((v_pool.permute(0, 3, 1, 2)[untouched] == 3.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("H, d, T", [(32, 64, 257), (3, 128, 2731), (5, 32, 1639)])
@pytest.mark.parametrize("activation, gate_first, per_row", [("sigmoid", False, False), ("silu", True, True)])
def test_gated_norm_of_many_rows(H, d, T, dtype, activation, gate_first, per_row):
    o = ops()
    g = torch.Generator("cuda").manual_seed(T + d)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, wide = randn(T, H * d), randn(H * d if per_row else d), randn(T, H * d + 16).to(dtype)
    gate, out = wide[:, 8:8 + H * d], torch.zeros(T, H * d + 8, dtype=dtype, device="cuda")
    o.gated_rmsnorm(x, w, gate, out[:, :H * d], H, d, 1e-5, activation, gate_first, 0.5)
    z = gate.double().view(T, H, d)
    act = torch.sigmoid(z) if activation == "sigmoid" else z * torch.sigmoid(z)
    v = x.double().view(T, H, d) * (act if gate_first else 1.0)
    want = v * torch.rsqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double().view(H if per_row else 1, d) * 0.5 * (1.0 if gate_first else act)
    tol = dict(rtol=2.0 ** -8, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=3e-6, atol=1e-6)
    torch.testing.assert_close(out[:, :H * d].double(), want.reshape(T, -1), **tol)
    assert not out[:, H * d:].any()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T, start, window, chunk", [(1024, 0, 100, 0), (1300, 77, 256, 0), (1025, 0, 1, 0), (2000, 3, 1000, 0), (1100, 60, 0, 300),
                                                     (1024, 0, 0, 128), (1500, 0, 4000, 0), (1400, 129, 129, 0)])
def test_windows_over_pairs_of_tiles(D, T, start, window, chunk):
    """Enough tiles that the kernel over pairs takes them: windows and runs of positions that begin and end anywhere in a block,
    shorter than a tile and longer than the sequence."""
    o = ops()
    H, G = 40, 8
    g = torch.Generator("cuda").manual_seed(T + window + chunk)
    kv = start + T
    W = -(-kv // 64)
    table = torch.randperm(W + 2, generator=torch.Generator().manual_seed(T))[:W].to(torch.int32).view(1, W).cuda()
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    q, k_pool, v_pool = randn(T, H * D), randn(W + 2, G, 64, D), randn(W + 2, G, D, 64)
    cu, kl = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.tensor([kv], dtype=torch.int32, device="cuda")
    out = torch.empty(T, H * D, dtype=torch.bfloat16, device="cuda")
    assert o.attention_prefill_tc(q, H * D, out, cu, kl, table, k_pool, v_pool, 1, T, H, G, D, window, chunk=chunk)
    assert o.attention_prefill_tc_status() == 0
    k = k_pool[table[0].long()].permute(1, 0, 2, 3).reshape(G, W * 64, D)[:, :kv].double()
    v = v_pool[table[0].long()].permute(1, 0, 3, 2).reshape(G, W * 64, D)[:, :kv].double()
    pos, key = torch.arange(start, kv, device="cuda")[:, None], torch.arange(kv, device="cuda")[None]
    hidden = (key > pos) | ((key < pos - pos % chunk) if chunk else (key <= pos - window))
    want = torch.empty(T, H, D, dtype=torch.float64, device="cuda")
    for h in range(H):
        s = (q[:, h * D:(h + 1) * D].double() @ k[h // 5].T / math.sqrt(D)).masked_fill(hidden, -math.inf)
        want[:, h] = s.softmax(-1) @ v[h // 5]
    # probabilities and results rounded to bfloat16: 2^-9 each of the values' unit spread, a little more where few keys are seen
    torch.testing.assert_close(out.double(), want.reshape(T, -1), rtol=2.0 ** -7, atol=2.0 ** -7)


@pytest.mark.parametrize("D, window, chunk", [(64, 1000, 0), (64, 0, 1024), (64, 300, 0), (128, 300, 0), (128, 0, 300), (128, 128, 0)])
def test_values_that_a_tile_does_not_read(D, window, chunk):
    """An infinite value reaches the rows whose tile of 128 reads its block of 128 keys, and no others: theirs are the bits without it.
    (Behind 200 positions the second tile of a pair starts up to eight blocks behind the first.)"""
    o = ops()
    H, G, T, start = 40, 8, 1300, 200
    kv = start + T
    g = torch.Generator("cuda").manual_seed(D + window + chunk)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    W = -(-kv // 64)
    table = torch.randperm(W, generator=torch.Generator().manual_seed(D)).to(torch.int32).view(1, W).cuda()
    q, k_pool, v_pool = randn(T, H * D), randn(W, G, 64, D), randn(W, G, D, 64)
    cu, kl = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.tensor([kv], dtype=torch.int32, device="cuda")

    def run(values):
        out = torch.empty(T, H * D, dtype=torch.bfloat16, device="cuda")
        assert o.attention_prefill_tc(q, H * D, out, cu, kl, table, k_pool, values, 1, T, H, G, D, window, chunk=chunk)
        assert o.attention_prefill_tc_status() == 0
        return out
    clean = run(v_pool)
    first = torch.tensor([start + r - r % 128 for r in range(T)])                  # position of the first row of a row's tile
    lowest = first - first % chunk if chunk else (first - window + 1).clamp(min=0)
    assert bool((lowest >= 128).any())
    for at in (10, 200, 400, 1023):
        poisoned = v_pool.clone()
        poisoned[int(table[0, at // 64]), :, :, at % 64] = math.inf
        got = run(poisoned)
        unread = (at // 128 < lowest // 128).cuda()
        assert torch.equal(got[unread], clean[unread])
        pos = torch.arange(start, kv)
        sees = (pos >= at) & ((at >= pos - pos % chunk) if chunk else (at > pos - window))
        assert not bool(got[sees.cuda()].isfinite().any())


@pytest.mark.parametrize("D, window, start", [(64, 1000, 1200), (64, 300, 500), (128, 300, 500), (128, 130, 1230), (128, 1, 192)])
def test_pages_that_a_window_has_let_go(D, window, start):
    """The table names page 0 in their place, which may hold anything of another sequence's: the bits with zeros in it."""
    o = ops()
    H, G, T = 40, 8, 1100
    kv = start + T
    gone = max(0, start - window + 1) // 64
    assert gone % 2 == 1                     # (the first block of 128 keys begins with a page that is gone)
    g = torch.Generator("cuda").manual_seed(D + window)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    W = -(-kv // 64)
    table = (1 + torch.randperm(W, generator=torch.Generator().manual_seed(D))).to(torch.int32).view(1, W).cuda()
    table[0, :gone] = 0
    q, k_pool, v_pool = randn(T, H * D), randn(W + 1, G, 64, D), randn(W + 1, G, D, 64)
    cu, kl = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.tensor([kv], dtype=torch.int32, device="cuda")
    outs = []
    for keys, values in ((0.0, 0.0), (math.nan, math.inf), (math.inf, math.nan)):
        k_pool[0], v_pool[0] = keys, values
        outs.append(torch.empty(T, H * D, dtype=torch.bfloat16, device="cuda"))
        assert o.attention_prefill_tc(q, H * D, outs[-1], cu, kl, table, k_pool, v_pool, 1, T, H, G, D, window)
        assert o.attention_prefill_tc_status() == 0
    assert bool(outs[0].isfinite().all()) and torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("G, a, b, D, T", [(1, 64, 32, 128, 300), (3, 40, 40, 96, 257), (2, 128, 64, 192, 2048)])
@pytest.mark.parametrize("turned", [False, True])
def test_key_rows_of_two_segments_of_many_tokens(G, a, b, D, T, turned, dtype):
    """A cached key row from two places of the projection (a normed part, then one that is turned or not and widened with zeros) and a value
    row: against the same launch in pieces of fewer tokens than the tile kernel takes, which differs in the order of the norm's sum."""
    o = ops()
    g = torch.Generator("cuda").manual_seed(T + D)
    raw = torch.randn(T, G * (2 * a + b) + 4, generator=g, device="cuda").to(dtype)
    weight = torch.randn(a, generator=g, device="cuda")
    W = -(-(T + 9) // 64)
    table = torch.randperm(W + 1, generator=torch.Generator().manual_seed(T))[:W].to(torch.int32).view(1, W).cuda()
    positions = torch.arange(9, T + 9, dtype=torch.int32, device="cuda")
    inv_freq = 1.0 / 10000.0 ** (torch.arange(b // 2, device="cuda").float() / (b // 2))
    seg = o.head_row_segment
    turn = {"half_pairs": b // 2, "turn_mul": 0.75} if turned else {}
    segments = o.head_row_segments(seg(4, G, a, 0, a, -1, True, 0, target=o.TO_CACHE_KEYS, cache_dim=D),
                                   seg(4 + G * a, G, b, a, D - a, mul=0.5, target=o.TO_CACHE_KEYS, cache_dim=D, **turn),
                                   seg(4 + G * (a + b), G, a, 0, D, target=o.TO_CACHE_VALUES))

    def run(piece):
        pools = [torch.full(s, 3.0, dtype=dtype, device="cuda") for s in ((W + 1, G, 64, D), (W + 1, G, D, 64))]
        for at in range(0, T, piece):
            part = slice(at, min(T, at + piece))
            pos = positions[part]
            o.head_rows(raw[part], None, segments, 1e-6, None, weight, cache=(pos, torch.zeros_like(pos), table, *pools),
                        rotary=(pos, inv_freq) if turned else None)
        return pools
    whole, pieces = run(T), run(100)
    assert torch.equal(whole[1], pieces[1])
    tol = dict(rtol=2.0 ** -7, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=2e-6, atol=2e-6)   # (one rounding to the type)
    torch.testing.assert_close(whole[0], pieces[0], **tol)
    page, at = table[0].long()[positions.long() // 64], positions.long() % 64
    first = raw[:, 4:4 + G * a].double().view(T, G, a)
    unit = first * torch.rsqrt((first * first).mean(-1, keepdim=True) + 1e-6) * weight.double()
    torch.testing.assert_close(whole[0][page, :, at, :a].double(), unit, **tol)
    assert not bool(whole[0][page, :, at, a + b:].any())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window, chunk", [(1000, 0), (777, 0), (0, 768), (0, 1000), (300, 0), (0, 130)])
@pytest.mark.parametrize("softcap, sink, gated", [(0.0, None, False), (2.0, 0.7, True), (0.0, 1.5, False), (30.0, None, True)])
def test_windows_with_terms_over_pairs_of_unequal_sequences(D, window, chunk, softcap, sink, gated):
    """Enough tiles for pairs of them (heads of 64 below 768 keys go a tile a CTA), sequences that end in a pair's first and second tile, behind nothing
    and behind prefixes that end inside a block."""
    o = ops()
    H, G, q_lens, behind = 20, 4, [700, 33, 1100], [0, 900, 77]
    kv = [q + b for q, b in zip(q_lens, behind)]
    g = torch.Generator("cuda").manual_seed(D + window + chunk)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    W, T = -(-max(kv) // 64), sum(q_lens)
    table = torch.randperm(3 * W + 1, generator=torch.Generator().manual_seed(D))[:3 * W].to(torch.int32).view(3, W).cuda()
    q, k_pool, v_pool = randn(T, H * D), randn(3 * W + 1, G, 64, D), randn(3 * W + 1, G, D, 64)
    gate = randn(T, H + 3)[:, :H]
    sinks = sink + 0.1 * torch.arange(H, device="cuda") if sink is not None else None
    cu = torch.tensor([0, 700, 733, T], dtype=torch.int32, device="cuda")
    out = torch.empty(T, H * D, dtype=torch.bfloat16, device="cuda")
    assert o.attention_prefill_tc(q, H * D, out, cu, torch.tensor(kv, dtype=torch.int32, device="cuda"), table, k_pool, v_pool, 3, max(q_lens), H, G, D,
                                  window, chunk=chunk, sinks=sinks, gate=gate if gated else None, softcap=softcap)
    assert o.attention_prefill_tc_status() == 0
    want = torch.empty(T, H, D, dtype=torch.float64, device="cuda")
    for s in range(3):
        k = k_pool[table[s].long()].permute(1, 0, 2, 3).reshape(G, W * 64, D)[:, :kv[s]].double()
        v = v_pool[table[s].long()].permute(1, 0, 3, 2).reshape(G, W * 64, D)[:, :kv[s]].double()
        pos, key = torch.arange(behind[s], kv[s], device="cuda")[:, None], torch.arange(kv[s], device="cuda")[None]
        hidden = (key > pos) | ((key < pos - pos % chunk) if chunk else (key <= pos - window))
        rows = slice(int(cu[s]), int(cu[s + 1]))
        for h in range(H):
            x = q[rows, h * D:(h + 1) * D].double() @ k[h * G // H].T / math.sqrt(D)
            x = (softcap * torch.tanh(x / softcap) if softcap else x).masked_fill(hidden, -math.inf)
            if sink is not None:
                x = torch.cat([x, sinks[h].double().expand(x.shape[0], 1)], 1)
            want[rows, h] = x.softmax(-1)[:, :kv[s]] @ v[h * G // H]
    if gated:
        want *= torch.sigmoid(gate.double())[:, :, None]
    # (probabilities and results rounded to bfloat16)
    torch.testing.assert_close(out.double(), want.reshape(T, -1), rtol=2.0 ** -7, atol=2.0 ** -7)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window, chunk", [(900, 0), (0, 1000), (0, 0)])
@pytest.mark.parametrize("counted", [False, True], ids=["shared out beforehand", "by counters"])
def test_pairs_of_tiles_on_two_streams(D, window, chunk, counted):
    """Launches without counters share nothing, and those with counters only with launches over the same ones: what two streams run at a
    time has the bits of each launch by itself, launch after launch, and the counters count the launches."""
    o = ops()
    H, G, T = 40, 8, 1500
    g = torch.Generator("cuda").manual_seed(D)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    W = -(-T // 64)
    table = torch.arange(W, dtype=torch.int32, device="cuda").view(1, W)
    q, k_pool, v_pool = randn(T, H * D), randn(W, G, 64, D), randn(W, G, D, 64)
    cu, kl = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.tensor([T], dtype=torch.int32, device="cuda")
    counters = torch.zeros(2, 4, dtype=torch.int32, device="cuda")

    def run(out, words):
        assert o.attention_prefill_tc(q, H * D, out, cu, kl, table, k_pool, v_pool, 1, T, H, G, D, window, chunk=chunk, work_counters=words)
    want, outs = torch.empty(T, H * D, dtype=torch.bfloat16, device="cuda"), torch.zeros(2, 20, T, H * D, dtype=torch.bfloat16, device="cuda")
    run(want, None)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for i in range(20):
        for out, stream, words in zip(outs, streams, counters):
            with torch.cuda.stream(stream):
                run(out[i], words if counted else None)
    torch.cuda.synchronize()
    assert o.attention_prefill_tc_status() == 0
    assert bool((outs == want).all())
    assert counters[:, 2:].tolist() == [[20, 0] if counted else [0, 0]] * 2
