"""Whole native calls (tensorrt_b200._native) against the general path, step by step through capi: the same bits for
every form they take, None for every other, and the errors of the general path unchanged."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _codes(b200, n, k, seed=0):
    w = (torch.randn(n, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)) * 0.02).bfloat16()
    return b200.capi.fp8_quantize(w, b200.capi.row_amax(w)), b200.capi.nvfp4_quantize(w, b200.capi.amax(w))


def _fp8_steps(capi, x, w, ws, bias, amax):
    xq, xs = capi.fp8_quantize(x, amax)
    return capi.fp8_gemm(xq, xs, w, ws, bias)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m", [1, 16, 40, 128, 129, 300])
def test_linears(b200, m, dtype):
    from tensorrt_b200 import _native

    capi, n, k = b200.capi, 520, 1056
    fp8, nv = _codes(b200, n, k)
    base = torch.randn(2, m, k + 32, device="cuda").to(dtype)
    bias = torch.randn(n, device="cuda").bfloat16()
    for x in (base[0, :, :k].contiguous(), base[:, :, :k], base[0, :, 32:]):          # plain, three dimensions and strided, offset
        rows = x.numel() // k
        for amax in (None, x.abs().max().float(), x.abs().amax(-1).float().reshape(-1)):
            for b in (None, bias):
                y = _native.fp8_linear(x, *fp8, b, amax, 0)
                assert y.dtype == torch.bfloat16 and torch.equal(y, _fp8_steps(capi, x, *fp8, b, amax))
                if amax is None or amax.numel() == 1:
                    ref = capi.nvfp4_gemm(*capi.nvfp4_quantize(x, capi.amax(x) if amax is None else amax), *nv, b)
                    assert torch.equal(_native.nvfp4_linear(x, *nv, b, amax, 0), ref)
        with capi.gemm_config(tile_n=128):
            assert torch.equal(b200.fp8_linear(x, *fp8), _fp8_steps(capi, x, *fp8, None, None))
        assert rows == x[..., 0].numel()
    assert capi.device_status() == 0


@pytest.mark.parametrize("m", [1, 48, 255, 256, 300])
@pytest.mark.parametrize("static_in,static_act", [(False, False), (True, False), (False, True), (True, True)])
def test_gated_mlp(b200, m, static_in, static_act, monkeypatch):
    from tensorrt_b200 import _native

    h, f = 272, 384
    g = torch.Generator(device="cuda").manual_seed(m)
    ws = [(torch.randn(*s, device="cuda", generator=g) * 0.05).bfloat16() for s in ((f, h), (f, h), (h, f))]
    x = torch.randn(m, h, device="cuda", generator=g).bfloat16()
    for per_channel in (True, False):
        mlp = b200.Fp8GatedMlp.from_float(*ws, per_channel=per_channel, input_amax=x.abs().max().float() if static_in else None,
                                          act_amax=torch.tensor(0.3, device="cuda") if static_act else None)
        y = _native.fp8_gated_mlp(x, mlp.gu_codes, mlp.gu_scales, mlp.down_codes, mlp.down_scales, mlp.input_amax, mlp.act_amax, 0)
        with monkeypatch.context() as mp:
            mp.setattr(_native, "fp8_gated_mlp", lambda *a: None)
            assert torch.equal(mlp(x), y)
        assert torch.equal(mlp(x), y)


def test_weights_written_just_before_the_call(b200):
    """A kernel that writes the weight codes directly in front of the call, itself launched under the tail of another:
    the GEMM requests weight tiles early and must still read the new ones."""
    from tensorrt_b200 import _lib

    capi, lib, n, k = b200.capi, _lib.load(), 8192, 8192
    ws = [(torch.randn(n, k, device="cuda") * 0.02).bfloat16() for _ in range(2)]
    quant = [capi.fp8_quantize(w, None) for w in ws]
    codes, scales = quant[0][0].clone(), quant[0][1].clone()
    st = torch.cuda.current_stream().cuda_stream
    for m in (1, 40, 128):
        x = torch.randn(m, k, device="cuda").bfloat16()
        refs = [_fp8_steps(capi, x, *q, None, None) for q in quant]
        torch.cuda.synchronize()
        for i in range(10):
            assert lib.b200q_fp8_quantize(ws[i & 1].data_ptr(), 2, n, k, None, 0, codes.data_ptr(), scales.data_ptr(), st) == 0
            y = b200.fp8_linear(x, codes, scales)
            assert torch.equal(y, refs[i & 1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m", [1, 2, 7, 16, 40])
def test_scales_and_bias_written_just_before_the_call(b200, m, dtype):
    """The same for the weight scales alone (the weights doubled: equal codes, other scales), for the bias, and for every
    part of an NVFP4 weight; m <= 16 FP8 tokens are one launch directly behind the writing kernel."""
    from tensorrt_b200 import _lib

    capi, lib, n, k = b200.capi, _lib.load(), 4096, 2048
    g = torch.Generator(device="cuda").manual_seed(m)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).bfloat16()
    ws, x = [w, w * 2], torch.randn(m, k, device="cuda", generator=g).to(dtype)
    zero, biases = torch.zeros(n, device="cuda").bfloat16(), [torch.randn(n, device="cuda", generator=g).bfloat16() for _ in range(2)]
    bias, st = biases[0].clone(), torch.cuda.current_stream().cuda_stream
    (codes, scales), (nc, ns, ng) = capi.fp8_quantize(w, None), capi.nvfp4_quantize(w, capi.amax(w))
    amax = [capi.amax(t).reshape(1) for t in ws]
    quant = [(capi.fp8_quantize(t, None), capi.nvfp4_quantize(t, a)) for t, a in zip(ws, amax)]
    assert torch.equal(quant[0][0][0], quant[1][0][0]) and not torch.equal(quant[0][0][1], quant[1][0][1])
    refs = []
    for (f8, nv), b in zip(quant, biases):
        refs.append((_fp8_steps(capi, x, *f8, b, None), capi.nvfp4_gemm(*capi.nvfp4_quantize(x, capi.amax(x)), *nv, b)))
    torch.cuda.synchronize()
    for i in range(10):
        f8_ref, nv_ref = refs[i & 1]
        assert lib.b200q_fp8_quantize(ws[i & 1].data_ptr(), 2, n, k, None, 0, codes.data_ptr(), scales.data_ptr(), st) == 0
        y_scales = b200.fp8_linear(x, codes, scales, biases[i & 1])
        capi.add(biases[i & 1], zero, out=bias)
        y_bias = b200.fp8_linear(x, codes, scales, bias)
        assert lib.b200q_nvfp4_quantize(ws[i & 1].data_ptr(), 2, n, k, amax[i & 1].data_ptr(), nc.data_ptr(), ns.data_ptr(), ng.data_ptr(), st) == 0
        y_nv = b200.nvfp4_linear(x, nc, ns, ng, biases[i & 1])
        assert torch.equal(y_scales, f8_ref) and torch.equal(y_bias, f8_ref) and torch.equal(y_nv, nv_ref)


def test_sdpa(b200):
    from tensorrt_b200 import _native

    q, k, v = (torch.randn(2, h, s, 48, device="cuda").half() for h, s in ((4, 130), (2, 77), (2, 77)))
    am = [t.abs().max().float() for t in (q, k, v)]
    for causal, scale in ((False, None), (True, None), (True, 0.2)):
        out = torch.empty_like(q)
        b200.capi._fp8_sdpa_into(out, q, k, v, *am, causal, scale)
        assert torch.equal(_native.fp8_sdpa(q, k, v, *am, causal, scale), out)
        assert torch.equal(_native.fp8_sdpa(q.transpose(1, 2).contiguous().transpose(1, 2), k, v, *am, causal, scale), out)


def test_other_inputs_take_the_general_path(b200):
    from torch._subclasses.fake_tensor import FakeTensorMode

    from tensorrt_b200 import _native

    capi = b200.capi
    (w, ws), _ = _codes(b200, 64, 64)
    x = torch.randn(3, 64, device="cuda").bfloat16()

    class Sub(torch.Tensor):
        pass

    for args in ((x.cpu(), w, ws, None, None), (x.double(), w, ws, None, None), (x[:, :48], w, ws, None, None), (x[:0], w, ws, None, None),
                 (x, w.t(), ws, None, None), (x, w, ws.double(), None, None), (x, w, ws[:5], None, None), (x, w, ws, ws, None),
                 (x, w, ws, None, torch.ones(2, device="cuda")), (x, w, ws, None, torch.ones(1)), (x.as_subclass(Sub), w, ws, None, None),
                 (x.to_sparse(), w, ws, None, None)):
        assert _native.fp8_linear(*args, 0) is None
    with FakeTensorMode():
        assert _native.fp8_linear(x, w, ws, None, None, 0) is None
    # what the general path accepts or refuses is unchanged
    assert torch.equal(b200.fp8_linear(x, w, ws, ws), _fp8_steps(capi, x, w, ws, ws, None))          # a bias of another type
    with pytest.raises(RuntimeError):
        b200.fp8_linear(x, w, ws, None, torch.ones(1))                                               # amax on the CPU
    with pytest.raises(ValueError):
        b200.fp8_linear(x, w, ws, None, torch.ones(2, device="cuda"))
    with pytest.raises(ValueError):
        b200.fp8_linear(x.double(), w, ws)
    with pytest.raises(RuntimeError):
        b200.fp8_linear(x.cpu(), w, ws)


def test_a_status_behind_the_first_launch_is_raised(b200):
    """A call whose later step is refused has already launched its quantize: it raises what the general path raises for it
    and does not go through that path from the start.  A call whose first step is refused returns None."""
    from tensorrt_b200 import _native

    def off8(t):                                                                                     # the same values, 8 bytes off
        return torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")[8:].view(t.shape).copy_(t)

    (w, ws), (nw, nws, ng) = _codes(b200, 256, 128)
    down, ds = _codes(b200, 128, 128)[0]
    for m in (1, 40):
        x = torch.randn(m, 128, device="cuda").bfloat16()
        for call in (lambda: _native.fp8_linear(x, off8(w), ws, None, None, 0), lambda: _native.nvfp4_linear(x, off8(nw), nws, ng, None, None, 0),
                     lambda: _native.fp8_gated_mlp(x, w, ws, off8(down), ds, None, None, 0), lambda: _native.fp8_linear(x, w, ws, None, None, 77)):
            with pytest.raises(b200.B200QError):
                call()
        shifted = torch.empty(m * 128 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(m, 128).copy_(x)
        assert _native.fp8_linear(shifted, w, ws, None, None, 0) is None and _native.nvfp4_linear(shifted, nw, nws, ng, None, None, 0) is None
    q, a = torch.randn(1, 2, 8, 16, device="cuda").bfloat16(), torch.ones(1, device="cuda")
    with pytest.raises(b200.B200QError):
        _native.fp8_sdpa(q, q, q, a, a, a, False, -1.0)
