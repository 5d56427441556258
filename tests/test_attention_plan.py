"""How a pass is attended by the kernels that take every size: into how many spans its keys are cut."""
from gpullama3.java_b200.kernels.ops import attention_paged_spans

SMS = 148


def test_spans_of_the_plain_kernel():
    for rows in (1, 2, 12, 32, 100, 200, 704, 1024, 1500, 4000, 5000, 100000):
        for reach in (1, 100, 128, 129, 500, 2000, 9000):
            spans, tiles = attention_paged_spans(rows, reach, SMS), -(-reach // 128)
            assert 1 <= spans <= min(16, tiles)
            chain = lambda n: -(-tiles // n) * -(-rows * n // (7 * SMS))
            assert spans == 1 or chain(spans) < chain(1)
    assert attention_paged_spans(32, 2000, SMS) == 16 and attention_paged_spans(32, 100, SMS) == 1
    assert attention_paged_spans(704, 2000, SMS) > 2 and attention_paged_spans(100000, 9000, SMS) == 1
