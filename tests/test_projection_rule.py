"""Which product takes a prompt's query/key/value projection with its rotation, without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from gpullama3.java_b200.kernels import fast, ops


@pytest.mark.parametrize("tokens, few_spans, spans, taken", [(45, 4, 1, "few"), (45, 4, 2, "few"), (45, 1, 1, "many"), (45, 1, 2, None),
                                                             (300, 4, 1, "many"), (300, 4, 2, None), (16, 4, 2, None)])
def test_angles_are_made_for_a_product_that_reads_them(monkeypatch, tokens, few_spans, spans, taken):
    seen = []
    monkeypatch.setattr(ops, "gemm_skinny_k_spans", lambda *a: few_spans, raising=False)
    monkeypatch.setattr(ops, "gemm_tcgen05_k_spans", lambda *a: spans)
    monkeypatch.setattr(ops, "gemm_skinny_qkv_rope", lambda x, *a: few_spans > 1 and (seen.append("few") or True))
    monkeypatch.setattr(ops, "gemm_tcgen05_qkv_rope", lambda *a: seen.append("many") or True)
    position = SimpleNamespace(rotary_dim=64, pairing=0, angles=lambda ctx: seen.append("angles"))
    mixer = SimpleNamespace(position=position, head_dim=64, n_heads=4, n_kv_heads=2)
    ctx = SimpleNamespace(all_decode=False, positions=None, seq_ids=None)
    x, w = torch.zeros(tokens, 128, dtype=torch.bfloat16), torch.zeros(512, 128, dtype=torch.bfloat16)
    assert fast.try_projection_with_rope(x, w, None, ctx, None, None, mixer, False) == (taken is not None)
    assert seen == (["angles", taken] if taken else [])
