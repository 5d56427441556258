"""Where float32 prompts are attended on the tensor cores: both sides of the rule as measured (32 heads of 64 over 8, 148 SMs)."""
import pytest

from gpullama3.java_b200.kernels.ops import _F32_TC_LAUNCHES, _F32_TC_PAGE, _attention_f32_fastest, attention_f32_tensor_cores_pay


@pytest.mark.parametrize("q_lens, behind, pays", [
    ([1024], [0], True), ([2048], [0], True), ([4096], [0], True), ([256] * 8, [0] * 8, True), ([512] * 4, [100] * 4, True),
    ([45], [0], False), ([256], [0], False), ([200], [1600], False), ([64], [2000], False), ([128], [4000], False),
    ([300, 17, 1, 700], [5, 900, 64, 0], False), ([16] * 16, [0] * 16, False)])
def test_rule_on_lengths(q_lens, behind, pays):
    kv_lens = [q + b for q, b in zip(q_lens, behind)]
    assert attention_f32_tensor_cores_pay(q_lens, kv_lens, 32, 8, 64, 148) == pays


def test_any_lengths_are_answered():
    """One-token sequences never pay; two prompts of 8,192 tokens do; and where the answer is yes, the other kernel is expected to take longer than
    three launches and one tile's walk over the longest sequence, which the rule's own figure cannot be below."""
    for n in (1, 2, 64):
        assert attention_f32_tensor_cores_pay([1] * n, [1] * n, 2, 1, 64, 148) is False
        assert attention_f32_tensor_cores_pay([1] * n, [5000] * n, 2, 1, 64, 148) is False
    assert attention_f32_tensor_cores_pay([8192] * 2, [8192] * 2, 32, 8, 64, 148) is True
    for q_lens, kv_lens in (([700, 5], [700, 900]), ([2048], [4096]), ([3] * 64, [3] * 64), ([16] * 100, [300] * 100)):
        other = _attention_f32_fastest(q_lens, kv_lens, 32, 8, 64, max(kv_lens), 148)[0]
        pays = attention_f32_tensor_cores_pay(q_lens, kv_lens, 32, 8, 64, 148)
        walk = _F32_TC_LAUNCHES + _F32_TC_PAGE * max(-(-k // 64) for k in kv_lens)      # (less than what the rule expects: one tile's pages)
        assert not pays or other > walk
