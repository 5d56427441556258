"""The float32 run's kernels at the sizes where they can go wrong: the product on the tensor cores (edges of its tiles,
cuts of K, every epilogue, rows off the 16-byte grid, sums that are not finite), the product for few rows, and the attention over tiles of queries."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -23


def ops():
    from gpullama3.java_b200.kernels import ops as o
    return o


def split_in_three(x):
    """The three bfloat16 parts of 2^24 x, in 64 bits."""
    x, parts = x.float() * 2.0 ** 24, []
    for _ in range(3):
        parts.append(x.to(torch.bfloat16).float())
        x = x - parts[-1]
    return [p.double() * 2.0 ** -24 for p in parts]


TERMS = [(2, 0), (0, 2), (1, 1), (1, 0), (0, 1), (0, 0)]
NORM = 3.0e-7      # of a product's errors; the kernel leaves 1.0e-7 to 1.3e-7 below K = 5,000
SHAPES = [(17, 64, 1024), (64, 128, 512), (129, 258, 1032), (300, 256, 4100), (100, 130, 2048)]


def operands(M, N, K):
    g = torch.Generator().manual_seed(M * N + K)
    return torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) / math.sqrt(K)


def _epilogue(o, epilogue, sums, c0, silu):
    if epilogue == o.EPILOGUE_STORE:
        out = sums.clone()
        out[:, :silu] = torch.nn.functional.silu(out[:, :silu])
        return out
    if epilogue == o.EPILOGUE_RESIDUAL_ADD:
        return c0.double() + sums
    g, u = sums[:, 0::2], sums[:, 1::2]
    if epilogue == o.EPILOGUE_GATED_SILU:
        return torch.nn.functional.silu(g) * u
    if epilogue == o.EPILOGUE_GATED_GELU_TANH:
        return torch.nn.functional.gelu(g, approximate="tanh") * u
    g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
    return g * torch.sigmoid(1.7 * g) * (u + 1)


@pytest.mark.parametrize("M, N, K, spans", [(17, 64, 1024, 0), (64, 128, 512, 0), (65, 130, 1028, 0), (129, 258, 1032, 0), (130, 1000, 68, 0),
                                            (300, 256, 4100, 0), (64, 300, 2048, 1), (200, 260, 1100, 3), (33, 514, 1024, 8)])
@pytest.mark.parametrize("epilogue", [0, 1, 2, 3, 4])
def test_products_on_the_tensor_cores_keep_32_bits(M, N, K, spans, epilogue):
    """A sum of K products has K / 64 float32 additions of partial sums, and within a partial sum at most 24 truncated ones:
    its error is below (K / 64 + 26) 2^-23 sum |a w| (two more for the terms left out and the bias).  The activations change
    a value by less than 1.5 times its argument's error here, and round a few times themselves."""
    o = ops()
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K + 5, generator=g).cuda()[:, 1:K + 1]                       # rows off the 16-byte grid, of another stride
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).cuda()
    bias = torch.randn(N, generator=g).cuda()
    columns = N // 2 if epilogue >= 2 else N
    c = torch.randn(M, columns + 3, generator=g).cuda()
    c0 = c.clone()
    silu = 37 if epilogue == 0 else 0
    assert o.gemm_f32_tcgen05(a, w, c[:, :columns], epilogue, (1.5, 1.7), bias, silu, n_spans=spans)
    sums = a.double() @ w.double().t() + bias.double()
    bound = (K / 64 + 26) * EPS * (a.double().abs() @ w.double().abs().t() + bias.abs().double())
    ref = _epilogue(o, epilogue, sums, c0[:, :columns], silu)
    if epilogue >= 2:
        big = sums.abs().amax() + 2
        bound = 1.5 * big * (bound[:, 0::2] + bound[:, 1::2]) + 16 * EPS * ref.abs()
    else:
        bound = 1.5 * bound + 16 * EPS * ref.abs()
    assert bool(((c[:, :columns].double() - ref).abs() <= bound).all())
    assert torch.equal(c[:, columns:], c0[:, columns:])
    assert o.gemm_f32_tcgen05_status() == 0


def test_products_whose_sums_are_not_finite():
    """Infinities and NaN come out where the plain product has them: such sums are formed again by multiply-adds."""
    o = ops()
    g = torch.Generator().manual_seed(3)
    a, w = torch.randn(100, 512, generator=g), torch.randn(200, 512, generator=g)
    a[3, 7], a[50, 100], w[20, 30], a[11, 5], w[5, 5] = math.inf, math.nan, -math.inf, 3.4e38, 1e-3
    a[60], a[61, 4] = math.nan, -3.39e38     # (the second rounds to an infinity as a bfloat16 number)
    a, w = a.cuda(), w.cuda()
    c = torch.empty(100, 200, device="cuda")
    assert o.gemm_f32_tcgen05(a, w, c)
    ref = torch.stack([o_row for o_row in (a.double().unsqueeze(1) * w.double().unsqueeze(0)).sum(-1)]).float()
    assert torch.equal(torch.isnan(c), torch.isnan(ref)) and torch.equal(torch.isinf(c), torch.isinf(ref))
    assert torch.equal(c[torch.isinf(c)], ref[torch.isinf(ref)])
    ok = torch.isfinite(ref)
    bound = 100 * EPS * (a.double().abs() @ w.double().abs().t())
    assert bool(((c.double() - ref.double()).abs()[ok] <= bound[ok]).all())
    assert o.gemm_f32_tcgen05_status() == 0


def test_products_that_stay_with_the_plain_kernels():
    o = ops()
    for M, N, K in ((16, 1024, 1024), (17, 1024, 1023), (17, 40, 2048), (100, 64, 64)):
        a, w, c = torch.zeros(M, K, device="cuda"), torch.zeros(N, K, device="cuda"), torch.full((M, N), 7.0, device="cuda")
        assert not o.gemm_f32_tcgen05(a, w, c) and bool((c == 7.0).all())
        o.gemm_generic(a, w, c)
        assert bool((c == 0).all())


@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 13, 16])
@pytest.mark.parametrize("N, K", [(8, 1024), (10, 1028), (130, 2048), (6, 4), (1002, 8192), (24, 3000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
def test_products_of_few_rows(M, N, K, dtype):
    """Below 4 + 5 + K / 1024 + 8 float32 additions to a sum, each of a half unit."""
    o = ops()
    g = torch.Generator().manual_seed(M * N + K)
    a, w = torch.randn(M, K, generator=g).to(dtype).cuda(), (torch.randn(N, K, generator=g) / math.sqrt(K)).to(dtype).cuda()
    bias = torch.randn(N, generator=g).cuda()
    ref = a.double() @ w.double().t() + bias.double()
    bound = (K / 1024 + 20) * EPS / 2 * (a.double().abs() @ w.double().abs().t() + bias.double().abs())
    c = torch.empty(M, N, device="cuda")
    o.gemm_generic(a, w, c, bias=bias)
    assert bool(((c.double() - ref).abs() <= bound).all())
    c0 = torch.randn(M, N, generator=g).cuda()
    c = c0.clone()
    o.gemm_generic(a, w, c, o.EPILOGUE_RESIDUAL_ADD, bias=bias)
    assert bool(((c.double() - c0.double() - ref).abs() <= bound + EPS * (c0.abs().double() + ref.abs())).all())
    h = torch.empty(M, N // 2, device="cuda")
    o.gemm_generic(a, w, h, o.EPILOGUE_GATED_SILU, bias=bias)
    gate, up = ref[:, 0::2], ref[:, 1::2]
    want = torch.nn.functional.silu(gate) * up
    slack = 1.2 * (bound[:, 0::2] * up.abs() + bound[:, 1::2] * gate.abs()) + 16 * EPS * want.abs() + 1e-9
    assert bool(((h.double() - want).abs() <= slack).all())


CUTS = [([5, 1, 100, 77], [5, 300, 100, 200]), ([70, 64, 65], [70, 64, 129]), ([130, 3], [400, 69])]


def attention_problem(q_lens, kv_lens, H, G, D, terms):
    """Queries, a paged cache that holds NaN behind every sequence's end, and the terms by name with their tensors."""
    terms = dict(terms)
    gen = torch.Generator("cuda").manual_seed(H * D)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    n, T, width = len(q_lens), sum(q_lens), max(-(-k // 64) for k in kv_lens)
    table = torch.randperm(n * width, generator=gen, device="cuda").to(torch.int32).view(n, width)
    k, v, q = rand(n * width, G, 64, D), rand(n * width, G, D, 64), rand(T, (H + 2 * G) * D) * 2
    biggest = float(v.abs().max())
    for i, length in enumerate(kv_lens):
        if length % 64:
            page = int(table[i, length // 64])
            k[page, :, length % 64:], v[page, :, :, length % 64:] = math.nan, math.nan
    if terms.pop("odd_values", 0):
        last = kv_lens[0] - 1
        v[int(table[0, last // 64]), :, 3, last % 64] = math.nan
        v[int(table[0, (last - 1) // 64]), :, 5, (last - 1) % 64] = math.inf
    window = terms.pop("window", 0)
    for name, shape in (("slopes", (H,)), ("sinks", (H,)), ("gate", (T, H + 3))):
        if terms.pop(name, 0):
            terms[name] = rand(*shape) * (0.1 if name == "slopes" else 1.0)
    positions = torch.cat([torch.arange(b - a, b) for a, b in zip(q_lens, kv_lens)]).to(torch.int32).cuda()
    seq_ids = torch.repeat_interleave(torch.arange(n), torch.tensor(q_lens)).to(torch.int32).cuda()
    cu = torch.tensor([0] + q_lens).cumsum(0).to(torch.int32).cuda()
    lens = torch.tensor(kv_lens, dtype=torch.int32, device="cuda")
    return q, k, v, table, positions, seq_ids, cu, lens, window, terms, biggest


def close_enough(got, want, D, biggest):
    """A score is a sum of D products of 2 normal numbers by normal numbers over sqrt(D): its rounding is below (D / 2 + 4) 2^-24 2 sqrt(D)
    on either side, and a result moves by at most twice that times the largest value."""
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    ok = torch.isfinite(want)
    assert float((got - want)[ok].abs().max()) <= 2 * 2 * (D / 2 + 4) * 2.0 ** -24 * 2 * math.sqrt(D) * biggest


@pytest.mark.parametrize("q_lens, kv_lens", CUTS)
@pytest.mark.parametrize("H, G, D", [(6, 2, 32), (4, 4, 64), (8, 1, 64), (6, 3, 96), (6, 2, 128)])
@pytest.mark.parametrize("terms", [{}, {"window": 33}, {"chunk": 48, "sinks": 1, "gate": 1}, {"slopes": 1, "softcap": 5.0, "window": 100, "sinks": 1},
                                   {"odd_values": 1}, {"odd_values": 1, "window": 20}], ids=str)
def test_attention_over_tiles_of_queries(q_lens, kv_lens, H, G, D, terms):
    """Against the plain kernel; with ``odd_values`` the last two positions of the first sequence hold values that are not finite,
    which earlier queries must not see."""
    o = ops()
    q, k, v, table, positions, seq_ids, cu, lens, window, terms, biggest = attention_problem(q_lens, kv_lens, H, G, D, terms)
    want, got = torch.empty(len(positions), H * D, device="cuda"), torch.full((len(positions), H * D), 7.0, device="cuda")
    o.attention_paged(q, q.shape[1], want, positions, seq_ids, table, k, v, H, G, D, window, **terms)
    assert o.attention_prefill_f32(q, q.shape[1], got, cu, lens, table, k, v, len(q_lens), max(q_lens), H, G, D, window, **terms)
    close_enough(got, want, D, biggest)


@pytest.mark.parametrize("kv_lens, n_spans", [([1, 64, 65, 300], 1), ([1, 64, 65, 300], 3), ([1030, 5], 16), ([700], 5)])
@pytest.mark.parametrize("H, G, D", [(6, 2, 32), (4, 4, 64), (8, 1, 64), (16, 1, 64), (12, 1, 96), (6, 2, 128)])
@pytest.mark.parametrize("terms", [{}, {"window": 33}, {"chunk": 48, "sinks": 1, "gate": 1}, {"slopes": 1, "softcap": 5.0, "window": 100, "sinks": 1},
                                   {"odd_values": 1}], ids=str)
def test_attention_of_decode_steps_in_spans(kv_lens, n_spans, H, G, D, terms):
    o = ops()
    q_lens = [1] * len(kv_lens)
    if terms.get("odd_values") and kv_lens[0] < 2:
        kv_lens = kv_lens[::-1]
    q, k, v, table, positions, seq_ids, cu, lens, window, terms, biggest = attention_problem(q_lens, kv_lens, H, G, D, terms)
    want, got = torch.empty(len(q_lens), H * D, device="cuda"), torch.full((len(q_lens), H * D), 7.0, device="cuda")
    o.attention_paged(q, q.shape[1], want, positions, seq_ids, table, k, v, H, G, D, window, **terms)
    assert o.attention_prefill_f32(q, q.shape[1], got, cu, lens, table, k, v, len(q_lens), 1, H, G, D, window, n_spans=n_spans, **terms)
    close_enough(got, want, D, biggest)


@pytest.mark.parametrize("q_lens, kv_lens", [([5, 1, 100, 77], [5, 300, 100, 500]), ([2], [1030]), ([3, 3, 1], [64, 65, 700])])
@pytest.mark.parametrize("H, G, D", [(6, 2, 32), (4, 4, 64), (16, 1, 64), (6, 3, 96), (6, 2, 128)])
@pytest.mark.parametrize("tile, n_spans", [(8, 1), (8, 5), (16, 3), (32, 1), (32, 16)])
@pytest.mark.parametrize("terms", [{}, {"chunk": 48, "sinks": 1, "gate": 1}, {"slopes": 1, "softcap": 5.0, "window": 100, "sinks": 1}, {"odd_values": 1}],
                         ids=str)
def test_attention_over_tiles_in_spans(q_lens, kv_lens, H, G, D, tile, n_spans, terms):
    """Tiles of every size, their keys whole and in spans (some of them empty), against the plain kernel."""
    o = ops()
    q, k, v, table, positions, seq_ids, cu, lens, window, terms, biggest = attention_problem(q_lens, kv_lens, H, G, D, terms)
    want, got = torch.empty(len(positions), H * D, device="cuda"), torch.full((len(positions), H * D), 7.0, device="cuda")
    o.attention_paged(q, q.shape[1], want, positions, seq_ids, table, k, v, H, G, D, window, **terms)
    assert o.attention_prefill_f32(q, q.shape[1], got, cu, lens, table, k, v, len(q_lens), max(q_lens), H, G, D, window, tile=tile, n_spans=n_spans,
                                   **terms)
    close_enough(got, want, D, biggest)


def attention_in_64_bits(q, k, v, table, q_lens, kv_lens, H, G, D):
    out, at = [], 0
    for i, (n, length) in enumerate(zip(q_lens, kv_lens)):
        pages = table[i, :-(-length // 64)].long()
        keys = k[pages].permute(0, 2, 1, 3).reshape(-1, G, D)[:length].double().repeat_interleave(H // G, 1)
        values = v[pages].permute(0, 3, 1, 2).reshape(-1, G, D)[:length].double().repeat_interleave(H // G, 1)
        s = torch.einsum("thd,jhd->htj", q[at:at + n, :H * D].double().view(n, H, D), keys) / math.sqrt(D)
        at += n
        hidden = torch.arange(length, device="cuda")[None, :] > torch.arange(length - n, length, device="cuda")[:, None]
        out.append(torch.einsum("htj,jhd->thd", s.masked_fill(hidden, -math.inf).softmax(-1), values).reshape(n, -1))
    return torch.cat(out)


@pytest.mark.parametrize("H, G, D", [(32, 8, 32), (32, 8, 64), (24, 8, 96), (24, 8, 128)])
@pytest.mark.parametrize("q_len, kv_len, tile, n_spans", [(300, 300, 32, 1), (200, 1800, 32, 1), (64, 2000, 32, 8), (16, 2000, 16, 16), (12, 1200, 8, 1)])
def test_attention_over_tiles_is_no_further_from_64_bits_than_the_plain_kernel(H, G, D, q_len, kv_len, tile, n_spans):
    """The norm of all errors (100,000 results and more, so that it moves by less than a fiftieth by chance) with every key unmasked where
    causality allows, queries as large as a norm leaves them."""
    o = ops()
    q, k, v, table, positions, seq_ids, cu, lens, _, _, _ = attention_problem([q_len], [kv_len], H, G, D, {})
    q /= 2
    want = attention_in_64_bits(q, k, v, table, [q_len], [kv_len], H, G, D)
    plain, got = torch.empty(q_len, H * D, device="cuda"), torch.empty(q_len, H * D, device="cuda")
    o.attention_paged(q, q.shape[1], plain, positions, seq_ids, table, k, v, H, G, D)
    assert o.attention_prefill_f32(q, q.shape[1], got, cu, lens, table, k, v, 1, q_len, H, G, D, tile=tile, n_spans=n_spans)
    assert float((got.double() - want).norm()) <= 1.02 * float((plain.double() - want).norm())


@pytest.mark.parametrize("q_lens, kv_lens", [([2], [700]), ([3, 1, 40], [3, 900, 40]), ([1] * 3, [900, 65, 1]), ([1] * 30, [500] * 30), ([150, 2], [150, 300])])
@pytest.mark.parametrize("H, G, D", [(8, 2, 64), (4, 4, 64), (6, 1, 128), (4, 2, 48)])
def test_attend_of_float32_passes(q_lens, kv_lens, H, G, D):
    """Through the choice of kernel, tile and spans that a model's mixers make; 48 has no tiles."""
    from types import SimpleNamespace

    from gpullama3.java_b200.parts.attention import attend

    q, k, v, table, positions, seq_ids, cu, lens, _, _, biggest = attention_problem(q_lens, kv_lens, H, G, D, {})
    for i, length in enumerate(kv_lens):      # (no NaN behind the ends: the plain computation here would meet them)
        if length % 64:
            page = int(table[i, length // 64])
            k[page, :, length % 64:], v[page, :, :, length % 64:] = 0.0, 0.0
    asked = []

    def empty(shape, dtype):
        asked.append(tuple(shape))
        return torch.empty(shape, dtype=dtype, device="cuda")

    ctx = SimpleNamespace(n_seqs=len(q_lens), q_lens=q_lens, start_pos=[b - a for a, b in zip(q_lens, kv_lens)], max_q_len=max(q_lens),
                          all_decode=max(q_lens) == 1, positions=positions, seq_ids=seq_ids, cu_seqlens=cu, kv_lens=lens, extras={}, scratch=empty,
                          capacity=lambda group: max(kv_lens))
    shape = SimpleNamespace(n_heads=H, n_kv_heads=G, head_dim=D, window=None, keep_first=0)
    out = torch.full((sum(q_lens), H * D), 7.0, device="cuda")
    attend(shape, q, out, ctx, table, SimpleNamespace(k=k, v=v, group=0))
    close_enough(out, attention_in_64_bits(q, k, v, table, q_lens, kv_lens, H, G, D).float(), D, biggest)
    if D != 48 and q_lens == [2]:
        assert ctx.extras and asked      # (two tokens behind 698: their keys go in spans, whose scratch the step gives)


@pytest.mark.parametrize("M", [64, 65, 100, 127, 128])
@pytest.mark.parametrize("N, K", [(1024, 64), (2050, 124), (512, 192), (512, 196)])
def test_products_of_a_short_k(M, N, K):
    """Tiles of 64 tokens up to 127 rows, of 128 from there and above K = 192."""
    o = ops()
    a, w = (t.cuda() for t in operands(M, N, K))
    c = torch.full((M, N), 7.0, device="cuda")
    assert o.gemm_f32_tcgen05(a, w, c)
    want = a.double() @ w.double().t()
    assert float((c.double() - want).norm() / want.norm()) < NORM


@pytest.mark.parametrize("M, N, K", SHAPES)
def test_every_term_of_a_product_is_there(M, N, K):
    """(Any one of the six missing: 2.2e-6 and more, test_float32_parts.py.)"""
    o = ops()
    a, w = (t.cuda() for t in operands(M, N, K))
    c = torch.empty(M, N, device="cuda")
    assert o.gemm_f32_tcgen05(a, w, c)
    want = a.double() @ w.double().t()
    assert float((c.double() - want).norm() / want.norm()) < NORM
    assert o.gemm_f32_tcgen05_status() == 0


@pytest.mark.parametrize("a_exponent, w_exponent", [(-100, 0), (-115, 20), (-125, 40), (-140, 60), (0, -105), (60, -122), (-60, -50), (60, -30)])
def test_products_of_small_numbers_keep_32_bits(a_exponent, w_exponent):
    """Down to subnormal numbers, whose bits the split must not lose either."""
    o = ops()
    a, w = operands(70, 200, 600)
    a, w = torch.ldexp(a, torch.tensor(float(a_exponent))).cuda(), torch.ldexp(w, torch.tensor(float(w_exponent))).cuda()
    c = torch.empty(70, 200, device="cuda")
    assert o.gemm_f32_tcgen05(a, w, c)
    want = a.double() @ w.double().t()
    assert float((c.double() - want).norm() / want.norm()) < NORM


@pytest.mark.parametrize("a_exponent, w_exponent", [(110, -90), (70, 20), (-30, 110), (60, 60)])
def test_products_of_large_numbers(a_exponent, w_exponent):
    """Numbers that leave no room for the scale and sums that leave none for its square are summed by multiply-adds: below K roundings."""
    o = ops()
    a, w = operands(40, 130, 600)
    a, w = torch.ldexp(a, torch.tensor(float(a_exponent))).cuda(), torch.ldexp(w, torch.tensor(float(w_exponent))).cuda()
    c = torch.empty(40, 130, device="cuda")
    assert o.gemm_f32_tcgen05(a, w, c)
    want = a.double() @ w.double().t()
    assert bool(torch.isfinite(c).all())
    assert bool(((c.double() - want).abs() <= 600 * EPS * (a.double().abs() @ w.double().abs().t())).all())


def test_a_float32_prompt_asks_nothing_of_the_allocator_once_its_workspace_fits(monkeypatch):
    """The split activations of the products and the spans of attention come from the pass's workspace; without memory to spare the products are
    made by multiply-adds and the keys are not cut."""
    from gpullama3.java_b200.engine.api import Engine, SequenceInput
    from gpullama3.java_b200.parts.base import StepContext

    config = {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": 2, "hidden_size": 256, "num_attention_heads": 4, "num_key_value_heads": 2,
              "head_dim": 64, "intermediate_size": 768, "vocab_size": 512, "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False,
              "max_position_embeddings": 1024}
    engine = Engine.from_random(config, 3, dtype="float32", max_tokens=64 * 12, max_batch=1)
    engine.step_fn.use_graphs = False

    def prompt():
        slot = engine.cache.acquire()
        engine.step([SequenceInput(slot, list(range(400)), [])])
        out = engine.step([SequenceInput(slot, list(range(20)), [19])])
        engine.cache.release(slot)
        return out.clone()

    want = prompt()
    prompt()
    asked, empty = [], torch.empty

    def counted(*args, **kwargs):
        t = empty(*args, **kwargs)
        if t.is_cuda:
            asked.append(t.numel())
        return t

    monkeypatch.setattr(torch, "empty", counted)
    assert torch.equal(prompt(), want)
    assert max(asked, default=0) <= want.numel()      # (the logits)
    monkeypatch.setattr(StepContext, "scratch", lambda self, shape, dtype: None)
    without = prompt()
    assert not torch.equal(without, want)
    torch.testing.assert_close(without, want, rtol=1e-4, atol=1e-4 * float(want.abs().max()))
