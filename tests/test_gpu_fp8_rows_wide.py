"""FP8 quantize and fake-quantize of 16-bit rows in 16-element pieces, at the edges of threads and pieces per thread, against
the kernel for unaligned rows (bases 16 bytes further on) and the oracle: the same codes, scales and values bit for bit, signed
zeros, a range below the data, and rows that are not finite included."""
import pytest
import torch

import oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [16, 512, 528, 4096, 4112, 5120, 8192, 8208, 14336, 16368, 16384])
def test_pieces_equal_groups(b200, cols, dtype):
    capi = b200.capi
    rows = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    g = torch.Generator(device="cuda").manual_seed(cols)
    wide = (torch.randn(rows, cols, device="cuda", generator=g) * 3).to(dtype)
    wide[1] = -0.0
    wide[2, ::3] = -0.0
    wide[3, cols - 1], wide[-1, 0] = float("nan"), float("-inf")
    store = torch.empty(rows * cols + 8, dtype=dtype, device="cuda")
    narrow = store[8:].view(rows, cols)
    narrow.copy_(wide)
    assert wide.data_ptr() % 32 == 0 and narrow.data_ptr() % 32 == 16
    same = lambda a, b: all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(a, b))  # noqa: E731
    row_amax = wide.float().abs().amax(1).nan_to_num(5.0, posinf=5.0)
    for amax in (None, torch.tensor(6.0, device="cuda"), torch.tensor(0.5, device="cuda"), torch.zeros((), device="cuda"), row_amax):
        assert same(capi.fp8_quantize(wide, amax), capi.fp8_quantize(narrow, amax))
    finite = wide[:3].cpu()
    codes, scales = capi.fp8_quantize(wide, None)
    c_ref, s_ref = o.fp8_quantize(finite, o.row_amax(finite))
    assert torch.equal(codes[:3].cpu(), c_ref) and torch.equal(scales[:3].cpu().view(-1, 1), s_ref)
    for amax in (6.0, 0.5):
        a = torch.tensor(amax)
        y = torch.ops.tensorrt.quantize_op(wide, a.cuda(), 8, 4, False, False)[:3]
        assert torch.equal(y.cpu().view(torch.int16), o.quantize_op(finite, a).view(torch.int16))
