"""The query/key/value product of a prompt of 17 to 128 tokens with rotation and cache write in its epilogue, against the product
followed by the rotation kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def ops():
    from gpullama3.java_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("H, KVH, D, M, K", [(32, 8, 64, 45, 2048), (24, 8, 128, 17, 3072), (32, 8, 128, 128, 4096), (4, 2, 64, 33, 512),
                                            (6, 2, 64, 100, 1000), (5, 1, 128, 64, 520), (32, 8, 64, 65, 520)])
@pytest.mark.parametrize("pairing", [0, 1], ids=["interleaved", "half"])
@pytest.mark.parametrize("write_cache", [True, False], ids=["writes", "reads_only"])
def test_few_token_projection_with_rotation_and_cache_write(H, KVH, D, M, K, pairing, write_cache):
    """Two sequences in one pass, the second behind 77 positions, pages scattered.  Both round the same sums to bfloat16 before they turn
    them by the same angles in the same order of roundings: the same bits, and what is not written is untouched."""
    o = ops()
    g = torch.Generator().manual_seed(H * D + M + pairing)
    N = (H + 2 * KVH) * D
    lens, starts = [M // 2, M - M // 2], [0, 77]
    positions = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, lens)]).to(torch.int32).cuda()
    seq_ids = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)]).to(torch.int32).cuda()
    width = max(-(-(s + n) // 64) for s, n in zip(starts, lens))
    n_pages = 2 * width + 3
    table = torch.randperm(n_pages, generator=g)[:2 * width].to(torch.int32).reshape(2, width).cuda()
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).to(torch.bfloat16).cuda()
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, D, 2).float() / D))).cuda()
    k0 = torch.randn(n_pages, KVH, 64, D, generator=g).to(torch.bfloat16).cuda()
    v0 = torch.randn(n_pages, KVH, D, 64, generator=g).to(torch.bfloat16).cuda()
    pools = lambda k, v: (k, v) if write_cache else (None, None)
    want, k_want, v_want = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), k0.clone(), v0.clone()
    assert o.gemm_skinny(a, w, want)
    o.rope_cache_write(want, positions, seq_ids, table, inv_freq, *pools(k_want, v_want), H, KVH, D, D, pairing, write_cache=write_cache)
    got, k_got, v_got = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda"), k0.clone(), v0.clone()
    assert o.gemm_skinny_qkv_rope(a, w, got, positions, seq_ids, table, o.rope_angles(positions, inv_freq, D // 2), *pools(k_got, v_got),
                                  H, KVH, D, pairing, write_cache)
    assert o.gemm_skinny_status() == 0
    assert torch.equal(v_got, v_want)
    assert torch.equal(got[:, :H * D], want[:, :H * D]) and torch.equal(k_got, k_want)
    assert bool((got[:, H * D:] == 7.0).all())
