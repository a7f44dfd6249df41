"""Residual add + RMSNorm + quantize at the edges of its launch shapes: one, two and four warps per row, the last column
count of each, rows at the threshold of the form and one past a CTA, bases that are 16-byte but not 32-byte aligned
(another kernel).  Codes and scales equal the separate kernels' bit for bit: the squares are added in the same order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("rows,cols", [(1184, 16), (1185, 48), (1187, 2032), (1184, 2048), (1191, 2064), (1185, 4080), (1184, 4096), (1187, 4112),
                                       (1185, 8192), (300, 8176), (1024, 4096), (2049, 1024)])
def test_matches_separate_kernels(b200, rows, cols, offset):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    make = lambda: torch.randn(rows * cols + offset, device="cuda", generator=g).bfloat16()[offset:].view(rows, cols)  # noqa: E731
    h, d = make(), make()
    h[3] = 0
    d[3] = -0.0
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=g)).bfloat16()
    for delta in (d, None):
        h_ref = capi.add(h, d) if delta is not None else h
        x = capi.rms_norm(h_ref, w)
        h_new, codes, scales = capi.add_rms_norm_fp8_quantize(h, delta, w)
        c_ref, s_ref = capi.fp8_quantize(x, None)
        assert torch.equal(h_new, h_ref) and torch.equal(codes, c_ref) and torch.equal(scales.flatten(), s_ref.flatten())
        for amax in (capi.amax(x), capi.amax(x) * 0.25):
            h_new, got = capi.add_rms_norm_nvfp4_quantize(h, delta, w, amax)
            ref = capi.nvfp4_quantize(x, amax)
            assert torch.equal(h_new, h_ref) and all(torch.equal(a, b) for a, b in zip(got, ref))
    assert capi.device_status() == 0


def test_rows_that_are_not_finite(b200):
    capi = b200.capi
    rows, cols = 1190, 4096
    h, d = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(2))
    h[0, cols // 2], h[1, 5], d[2, cols - 1] = float("nan"), float("inf"), float("nan")
    w = torch.ones(cols, device="cuda").bfloat16()
    x = capi.rms_norm(capi.add(h, d), w)
    _, codes, scales = capi.add_rms_norm_fp8_quantize(h, d, w)
    c_ref, s_ref = capi.fp8_quantize(x, None)
    assert torch.equal(codes, c_ref) and torch.equal(scales.flatten(), s_ref.flatten())
    amax = torch.tensor(4.0, device="cuda")
    got, ref = capi.add_rms_norm_nvfp4_quantize(h, d, w, amax)[1], capi.nvfp4_quantize(x, amax)
    assert all(torch.equal(a, b) for a, b in zip(got, ref))


@pytest.mark.parametrize("rows,cols", [(1, 2048), (3, 2064), (17, 16384), (33, 10240), (147, 4112), (295, 2048)])
def test_few_rows_one_piece_per_thread(b200, rows, cols):
    """A CTA per row adds the squares in an order of its own: the last bits of the sum move rsqrt and the products by up to 2
    ulp of fp32, which changes one in 2^14 bf16 roundings at most, and with it a code (or, through a row's abs-max, a scale)."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    h, d = (torch.randn(rows, cols, device="cuda", generator=g).bfloat16() for _ in range(2))
    h[rows // 2] = 0
    d[rows // 2] = -0.0
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=g)).bfloat16()
    few = lambda a, b: int((a != b).sum()) <= max(1, b.numel() >> 13)  # noqa: E731
    for delta in (d, None):
        h_ref = capi.add(h, d) if delta is not None else h
        x = capi.rms_norm(h_ref, w)
        h_new, codes, scales = capi.add_rms_norm_fp8_quantize(h, delta, w)
        c_ref, s_ref = capi.fp8_quantize(x, None)
        same = scales.flatten() == s_ref.flatten()
        assert torch.equal(h_new, h_ref) and int((~same).sum()) <= 1 + rows // 64 and few(codes[same], c_ref[same])
        amax = capi.amax(x)
        h_new, got = capi.add_rms_norm_nvfp4_quantize(h, delta, w, amax)
        ref = capi.nvfp4_quantize(x, amax)
        assert torch.equal(h_new, h_ref) and torch.equal(got[2], ref[2]) and all(few(a, b) for a, b in zip(got[:2], ref[:2]))
    assert capi.device_status() == 0


@pytest.mark.parametrize("with_delta", [True, False])
@pytest.mark.parametrize("rows,cols", [(5, 4096), (1190, 4096), (1190, 528)])
def test_nan_beside_values_above_the_range(b200, rows, cols, with_delta):
    """A NaN norm weight puts one NaN into a block of every row; under a range far below the data the block's scale saturates
    and the NaN's code is decided there.  Small integers in: the sum of squares is the same in any order, codes are compared
    bit for bit."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    h, d = (torch.randint(-3, 4, (rows, cols), device="cuda", generator=g).bfloat16() for _ in range(2))
    w = torch.ones(cols, device="cuda").bfloat16()
    w[5], w[cols - 1] = float("nan"), -float("nan")
    delta = d if with_delta else None
    x = capi.rms_norm(capi.add(h, d) if with_delta else h, w)
    assert bool(x[:, 5].isnan().all())
    for amax in (0.25, 4.0):
        amax = torch.tensor(amax, device="cuda")
        got, ref = capi.add_rms_norm_nvfp4_quantize(h, delta, w, amax)[1], capi.nvfp4_quantize(x, amax)
        assert all(torch.equal(a, b) for a, b in zip(got, ref))


@pytest.mark.parametrize("rows,cols,offset", [(5, 2064, 8), (200, 8192, 8), (200, 16384, 8), (64, 4096, 8), (80, 12288, 8), (5, 8192, 8),
                                              (16, 16384, 0), (7, 2048, 0), (64, 8192, 0), (200, 4112, 0)])
@pytest.mark.parametrize("finite", [True, False])
def test_few_rows_of_small_integers(b200, rows, cols, offset, finite):
    """Few rows on clusters of two (one, two and four groups of 8 a thread), four (one, two) and eight CTAs, which take bases 16
    but not 32 bytes aligned, on clusters of eight with aligned bases, and on a CTA per row.  Small integers: the sum of squares
    is the same in any order, so codes and scales equal the separate kernels' bit for bit, a range below the data included."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    make = lambda: torch.randint(-3, 4, (rows * cols + offset,), device="cuda", generator=g).bfloat16()[offset:].view(rows, cols)  # noqa: E731
    h, d = make(), make()
    h[rows // 2] = 0
    d[rows // 2] = -0.0
    if not finite:
        h[0, cols // 2], h[1, 5], d[2, cols - 1] = float("nan"), float("inf"), float("nan")
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=g)).bfloat16()
    same = lambda a, b: torch.equal(a.flatten().view(torch.uint8), b.flatten().view(torch.uint8))  # noqa: E731
    for delta in (d, None):
        h_ref = capi.add(h, d) if delta is not None else h
        x = capi.rms_norm(h_ref, w)
        h_new, codes, scales = capi.add_rms_norm_fp8_quantize(h, delta, w)
        c_ref, s_ref = capi.fp8_quantize(x, None)
        assert same(h_new, h_ref) and same(codes, c_ref) and same(scales, s_ref)
        for amax in (4.0, 0.5):
            amax = torch.tensor(amax, device="cuda")
            got, ref = capi.add_rms_norm_nvfp4_quantize(h, delta, w, amax)[1], capi.nvfp4_quantize(x, amax)
            assert all(torch.equal(a, b) for a, b in zip(got, ref))
    assert capi.device_status() == 0
