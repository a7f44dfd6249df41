"""FP8 quantize and fake-quantize of many 16-bit rows of 2049 to 3072 elements, which go in 16-element pieces as shorter and longer rows
do: bit for bit the kernel for unaligned rows (bases 16 bytes further on), on both sides of the limits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [2048, 2064, 2560, 3056, 3072, 3088])
def test_pieces_equal_groups(b200, cols, dtype):
    capi = b200.capi
    rows = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    g = torch.Generator(device="cuda").manual_seed(cols)
    wide = (torch.randn(rows, cols, device="cuda", generator=g) * 3).to(dtype)
    wide[1, ::3] = -0.0
    wide[2, cols - 1], wide[-1, 0], wide[3, 7] = float("nan"), float("-inf"), 6e4
    narrow = torch.empty(rows * cols + 8, dtype=dtype, device="cuda")[8:].view(rows, cols).copy_(wide)
    assert wide.data_ptr() % 32 == 0 and narrow.data_ptr() % 32 == 16
    bits = lambda t: t.view(torch.uint8)  # noqa: E731
    for amax in (None, torch.tensor(6.0, device="cuda"), torch.tensor(0.5, device="cuda"), torch.full((rows,), 2.0, device="cuda")):
        for a, b in zip(capi.fp8_quantize(wide, amax), capi.fp8_quantize(narrow, amax)):
            assert torch.equal(bits(a), bits(b))
        if amax is not None and amax.numel() == 1:
            assert torch.equal(bits(capi.fp8_fake_quantize(wide, amax)), bits(capi.fp8_fake_quantize(narrow, amax)))
