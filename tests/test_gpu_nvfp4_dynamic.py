"""NVFP4 quantize under the measured abs-max: codes, swizzled scales and global scale equal abs-max and quantize run one
after the other, on both sides of the size where one launch takes over, and with rows that are not whole scale words."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 16), (1, 4096), (3, 80), (16, 8192), (16, 8208), (127, 1024), (128, 1024), (129, 1024), (8192, 16),
                                       (2, 28672), (1, 131072), (1, 131088), (16, 4096), (16, 4112), (1, 65536), (1, 65600), (129, 512)])
def test_dynamic(b200, rows, cols, dtype):
    capi = b200.capi
    x = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows + cols)).to(dtype)
    for t in (x, torch.zeros_like(x)):
        for a, b in zip(capi.nvfp4_quantize_dynamic(t), capi.nvfp4_quantize(t, capi.amax(t))):
            assert a.shape == b.shape and torch.equal(a, b)
