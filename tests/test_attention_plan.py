"""How a float32 pass is attended: the choice of tile and spans, for every kind of pass that the engine makes."""
import itertools

import pytest

from gpullama3.java_b200.kernels.ops import PAGE_TOKENS, attention_f32_plan, attention_paged_spans

SMS = 148


@pytest.mark.parametrize("H, G, D", [(32, 8, 64), (32, 32, 64), (16, 1, 128), (12, 6, 32), (24, 8, 96), (40, 1, 64)])
def test_plans_are_ones_that_the_kernels_take(H, G, D):
    for n, q, behind in itertools.product((1, 3, 64, 500), (1, 2, 5, 17, 64, 300, 4000), (0, 1, 63, 500, 9000)):
        if n * q > 20000:
            continue
        kv = behind + q
        for reach in {kv, min(kv, 100), 1}:
            tile, spans = attention_f32_plan([q] * n, [kv] * n, H, G, D, reach, SMS)
            assert (tile, spans) == (0, 0) and H // G <= 2 or tile in (8, 16, 32) and 1 <= spans <= min(16, -(-reach // PAGE_TOKENS))


def ctas(q_lens, H, G, tile, spans):
    return sum(-(-q * (H // G) // tile) for q in q_lens) * G * spans


@pytest.mark.parametrize("q", [2, 4, 8, 16])
@pytest.mark.parametrize("behind", [2000, 8000])
def test_few_tokens_behind_a_long_context_fill_the_gpu(q, behind):
    tile, spans = attention_f32_plan([q], [behind + q], 32, 8, 64, behind + q, SMS)
    assert tile * 2 <= max(16, 4 * q) * 2 and ctas([q], 32, 8, tile, spans) >= 0.8 * SMS


def test_sequences_that_decode_beside_a_prompt_are_cut_into_spans():
    q_lens, kv_lens = [40] + [1] * 8, [40] + [2000] * 8
    tile, spans = attention_f32_plan(q_lens, kv_lens, 32, 8, 64, 2000, SMS)
    assert spans >= 2 and ctas(q_lens, 32, 8, tile, spans) >= 2 * SMS


def test_long_prompts_take_large_tiles_without_spans():
    assert attention_f32_plan([2048], [2048], 32, 8, 64, 2048, SMS) == (32, 1)
    assert attention_f32_plan([512] * 8, [512] * 8, 32, 8, 128, 512, SMS) == (32, 1)


def test_one_head_to_a_kv_head_decodes_row_by_row():
    assert attention_f32_plan([1] * 8, [2000] * 8, 32, 32, 64, 2000, SMS) == (0, 0)
    assert attention_f32_plan([1] * 8, [2000] * 8, 32, 8, 64, 2000, SMS)[0] == 8


def test_spans_of_the_plain_kernel():
    for rows in (1, 2, 12, 32, 100, 200, 704, 1024, 1500, 4000, 5000, 100000):
        for reach in (1, 100, 128, 129, 500, 2000, 9000):
            spans, tiles = attention_paged_spans(rows, reach, SMS), -(-reach // 128)
            assert 1 <= spans <= min(16, tiles)
            chain = lambda n: -(-tiles // n) * -(-rows * n // (7 * SMS))
            assert spans == 1 or chain(spans) < chain(1)
    assert attention_paged_spans(32, 2000, SMS) == 16 and attention_paged_spans(32, 100, SMS) == 1
    assert attention_paged_spans(704, 2000, SMS) > 2 and attention_paged_spans(100000, 9000, SMS) == 1
