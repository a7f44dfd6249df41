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
