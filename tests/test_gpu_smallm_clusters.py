"""Small-M GEMM at the weight shapes where the cluster size changes: just below, at and above the tile counts that clusters of
eight and four are resident for, short K.  Operands are small integers, so that every order of summation gives the same fp32
value and the result is compared bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 17, 33, 64, 128])
@pytest.mark.parametrize("N,K", [(1024, 128), (1536, 2048), (1664, 2048), (2048, 2048), (2304, 1040), (4224, 1536), (4352, 1536), (4608, 1536), (6144, 512)])
def test_fp8_cluster_sizes(b200, tokens, N, K):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(tokens + N + K)
    x = torch.randint(-2, 3, (tokens, K), device="cuda", generator=g).float()
    w = torch.randint(-2, 3, (N, K), device="cuda", generator=g).float()
    to_codes = lambda t: t.to(torch.float8_e4m3fn).view(torch.uint8)  # noqa: E731
    y = capi.fp8_gemm(to_codes(x), torch.ones(tokens, device="cuda"), to_codes(w), torch.ones(N, device="cuda"))
    ref = (x.double() @ w.double().t()).bfloat16()
    assert torch.equal(y, ref)
    assert capi.device_status() == 0


@pytest.mark.parametrize("tokens", [1, 33, 128])
@pytest.mark.parametrize("N,K", [(1536, 4096), (1920, 2048), (2048, 2048), (4224, 2048), (4352, 2048), (9088, 1056), (9216, 1056), (9472, 1056)])
def test_nvfp4_cluster_sizes(b200, tokens, N, K):
    """The same at 12, 15, 16, 33, 34, 71, 72 and 74 tiles in NVFP4: E2M1 codes of small integers under scales of one."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(tokens + N + K)
    values = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device="cuda")

    def operand(rows):
        codes = torch.randint(0, 5, (rows, K), device="cuda", generator=g) + 8 * torch.randint(0, 2, (rows, K), device="cuda", generator=g)
        ref = values[codes & 7] * torch.where(codes >= 8, -1.0, 1.0)
        scales = torch.full(((rows + 127) // 128 * 128 * ((K // 16 + 3) // 4 * 4),), 0x38, dtype=torch.uint8, device="cuda")
        return ((codes[:, 0::2] | (codes[:, 1::2] << 4)).to(torch.uint8), scales, torch.ones(1, device="cuda")), ref

    (xq, x), (wq, w) = operand(tokens), operand(N)
    y = capi.nvfp4_gemm(*xq, *wq)
    assert torch.equal(y, (x.double() @ w.double().t()).bfloat16())
    assert capi.device_status() == 0
