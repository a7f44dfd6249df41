"""Kernels that quantize to NVFP4 what they produce (residual add + RMSNorm, silu(gate) * up, repeated kv heads) under a
calibrated amax: codes, swizzled scales (padding rows included) and global scale equal the separate kernels' bit for
bit, at row counts around 128-row scale tiles and at the edges of their launch shapes.  With few long rows the norm adds the
squares in another order; codes may then differ as rarely as a bf16 rounding does."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _same(got, ref):
    for a, b in zip(got, ref):
        assert a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("with_delta", [True, False])
@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 272), (5, 4096), (64, 8192), (127, 2064), (128, 2048), (300, 4096), (1184, 4096),
                                       (1300, 2080), (1190, 8192), (2, 16384), (400, 16384)])
def test_add_rms_norm(b200, rows, cols, with_delta):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    h, d = (torch.randn(rows, cols, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=g)).bfloat16()
    delta = d if with_delta else None
    h_ref = capi.add(h, d) if with_delta else h
    x = capi.rms_norm(h_ref, w)
    split = rows < 2 * torch.cuda.get_device_properties(0).multi_processor_count and cols >= 2048     # few long rows
    for amax in (capi.amax(x), capi.amax(x) * 0.25, torch.zeros((), device="cuda")):
        h_new, got = capi.add_rms_norm_nvfp4_quantize(h, delta, w, amax)
        assert torch.equal(h_new, h_ref)
        ref = capi.nvfp4_quantize(x, amax)
        if split:
            # the sum's last bits move rsqrt and the products by up to 2 ulp of fp32, one in 2^14 bf16 roundings at most
            assert torch.equal(got[2], ref[2])
            assert all(int((a != b).sum()) <= max(1, b.numel() >> 13) for a, b in zip(got[:2], ref[:2]))
        else:
            _same(got, ref)
    assert capi.device_status() == 0


def _scales_by_row(sf, cols):
    """Swizzled scales -> [rows padded to 128, columns padded to 64 / 16]."""
    tiles = sf.view(-1, (cols // 16 + 3) // 4, 32, 4, 4)                # [row tile, column tile, row % 32, row // 32 % 4, 4 scales]
    return tiles.permute(0, 3, 2, 1, 4).reshape(-1, tiles.shape[1] * 4)


@pytest.mark.parametrize("rows,cols", [(3, 272), (5, 4096), (300, 4096), (1300, 2080)])      # CTAs of 8-element groups, a CTA a row of 16-element pieces, groups again, warps
def test_add_rms_norm_of_rows_that_are_not_finite(b200, rows, cols):
    """A NaN makes its whole row NaN, an infinity makes its row zeros with one NaN: as the separate kernels store them."""
    capi = b200.capi
    h, d = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(2))
    h[0, cols // 2], h[1, 5], d[2, cols - 1] = float("nan"), float("inf"), float("nan")
    w = torch.ones(cols, device="cuda").bfloat16()
    x = capi.rms_norm(capi.add(h, d), w)
    amax = torch.tensor(4.0, device="cuda")
    _, (codes, sf, _) = capi.add_rms_norm_nvfp4_quantize(h, d, w, amax)
    ref_codes, ref_sf, _ = capi.nvfp4_quantize(x, amax)
    sf, ref_sf = _scales_by_row(sf, cols), _scales_by_row(ref_sf, cols)
    assert torch.equal(codes[:3], ref_codes[:3]) and torch.equal(sf[:3], ref_sf[:3])
    assert int(sf[0, :cols // 16].min()) == int(sf[2, :cols // 16].min()) == 0x7F and int(sf[1].max()) == 0


@pytest.mark.parametrize("rows,f", [(1, 16), (3, 528), (128, 1040), (130, 14336), (33, 28672)])
def test_silu_mul(b200, rows, f):
    capi = b200.capi
    gu = torch.randn(rows, 2 * f, device="cuda", generator=torch.Generator(device="cuda").manual_seed(f)).bfloat16() * 3
    act = capi.silu_mul(gu)
    for amax in (capi.amax(act), capi.amax(act) * 0.3):
        _same(capi.silu_mul_nvfp4_quantize(gu, amax), capi.nvfp4_quantize(act, amax))


@pytest.mark.parametrize("rows,n_q,n_kv,d", [(1, 2, 1, 16), (5, 8, 2, 48), (129, 32, 8, 128), (64, 16, 8, 64)])
def test_expand_heads(b200, rows, n_q, n_kv, d):
    capi = b200.capi
    qkv = torch.randn(rows, (n_q + 2 * n_kv) * d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(d)).bfloat16()
    col0, rep = (n_q + n_kv) * d, n_q // n_kv
    wide = capi.expand_heads(qkv, col0, n_q, rep, d)
    amax = capi.amax(wide)
    _same(capi.expand_heads_nvfp4_quantize(qkv, col0, n_q, rep, d, amax), capi.nvfp4_quantize(wide, amax))


@pytest.mark.parametrize("rows", [1, 16, 127, 128, 129, 300])
def test_padding_rows_of_the_scale_tile_are_cleared(b200, rows):
    from tensorrt_b200 import _lib

    cols = 80
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    amax = x.abs().max().float().reshape(1)
    codes, ref, g = b200.capi.nvfp4_quantize(x, amax)
    sf = torch.full_like(ref, 0xAA)
    assert _lib.load().b200q_nvfp4_quantize(x.data_ptr(), 2, rows, cols, amax.data_ptr(), codes.data_ptr(), sf.data_ptr(), g.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream) == 0
    by_row = _scales_by_row(sf, cols)
    assert int(by_row[rows:].max() if by_row.shape[0] > rows else 0) == 0
    assert int(by_row[:rows, cols // 16:].max()) == 0 and bool((by_row[:rows, :cols // 16] != 0xAA).all())
