"""FP8 attention at the edges of its key tiles: one to five tiles of 128 keys (the score pipeline holds two in flight),
whole and ragged last tiles, causal edges, and the head dimensions at which the contraction takes fewer steps.
Tolerance as in test_gpu_attention: rel-L2 <= 1e-2 against the oracle (same quantization points)."""
import pytest
import torch

import oracle as o


@pytest.mark.gpu
@pytest.mark.parametrize("D", [16, 80, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("sk", [1, 127, 128, 129, 256, 257, 384, 511, 640])
def test_key_tile_edges(b200, sk, causal, D):
    g = torch.Generator().manual_seed(sk + D)
    sq = sk if causal else 130
    q = (torch.randn(1, 2, sq, D, generator=g) * 1.5).bfloat16()
    k = (torch.randn(1, 1, sk, D, generator=g) * 1.5).bfloat16()
    v = torch.randn(1, 1, sk, D, generator=g).bfloat16()
    aq, ak, av = (t.float().abs().max() for t in (q, k, v))
    ref = o.fp8_sdpa_ref(q, k, v, aq, ak, av, is_causal=causal)
    out = b200.capi.fp8_sdpa(q.cuda(), k.cuda(), v.cuda(), aq.cuda(), ak.cuda(), av.cuda(), is_causal=causal)
    torch.cuda.synchronize()
    assert b200.capi.device_status() == 0
    assert o.rel_l2(out.float().cpu(), ref.float()) <= 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,sq,causal", [(42, 42, 130, False), (42, 42, 300, True), (80, 40, 129, True)])
def test_head_groups(b200, hq, hkv, sq, causal):
    """Heads whose keys and values do not fit L2 are walked in groups (32 kv heads of 4096 x 128 here, the last group smaller):
    the same bits as a call per head, which is one group."""
    g = torch.Generator(device="cuda").manual_seed(hq)
    q, k, v = (torch.randn(1, h, s, 128, device="cuda", generator=g).bfloat16() for h, s in ((hq, sq), (hkv, 4096), (hkv, 4096)))
    a = torch.tensor(4.0, device="cuda")
    out = b200.capi.fp8_sdpa(q, k, v, a, a, a, is_causal=causal)
    for h in range(hq):
        n = h // (hq // hkv)
        one = b200.capi.fp8_sdpa(q[:, h:h + 1], k[:, n:n + 1], v[:, n:n + 1], a, a, a, is_causal=causal)
        assert torch.equal(out[:, h:h + 1], one)
    assert b200.capi.device_status() == 0
