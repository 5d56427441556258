"""Where float32 prompts are attended on the tensor cores: both sides of the rule as measured (32 heads of 64 over 8, 148 SMs)."""
import pytest

from gpullama3.java_b200.kernels.ops import attention_f32_tensor_cores_pay


@pytest.mark.parametrize("q_lens, behind, pays", [
    ([1024], [0], True), ([2048], [0], True), ([4096], [0], True), ([256] * 8, [0] * 8, True), ([512] * 4, [100] * 4, True),
    ([45], [0], False), ([256], [0], False), ([200], [1600], False), ([64], [2000], False), ([128], [4000], False),
    ([300, 17, 1, 700], [5, 900, 64, 0], False), ([16] * 16, [0] * 16, False)])
def test_rule_on_lengths(q_lens, behind, pays):
    kv_lens = [q + b for q, b in zip(q_lens, behind)]
    assert attention_f32_tensor_cores_pay(q_lens, kv_lens, 32, 8, 64, 148) == pays


def test_any_lengths_are_answered():
    for q_lens, kv_lens in (([1], [1]), ([1, 1], [5000, 1]), ([8192] * 2, [8192] * 2), ([3] * 64, [3] * 64)):
        assert attention_f32_tensor_cores_pay(q_lens, kv_lens, 2, 1, 64, 148) in (True, False)
