"""A forward of the decoder stack as one native call against the same forward issued call by call: the same bits, for both formats, both
attention cores, and on either side of every choice of kernel on the way; and what the native call leaves to the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stack(b200, mode, n_q, n_kv, hd, ffn, layers, seq_len, calibrate):
    from tensorrt_b200.stack import DecoderStack, StackConfig, random_layer_weights

    cfg = StackConfig(hidden=n_q * hd, n_q=n_q, n_kv=n_kv, head_dim=hd, ffn=ffn, layers=layers, mode=mode,
                      attention="fp8_sdpa" if seq_len else "identity", seq_len=seq_len)
    stack = DecoderStack(cfg, random_layer_weights(cfg, 3))
    if calibrate:
        stack.calibrate(torch.randn(max(seq_len, 64), cfg.hidden, device="cuda").bfloat16())
    return stack


def _by_calls(stack, h):
    stack.native_layers = False
    try:
        return stack.forward(h)
    finally:
        stack.native_layers = True


@pytest.mark.parametrize("tokens", [1, 64, 130, 255, 256, 520])
@pytest.mark.parametrize("mode,n_q,n_kv,hd,ffn,seq_len", [
    ("fp8", 4, 2, 64, 768, 0),          # activation in the GEMM's epilogue from 256 tokens on
    ("fp8", 4, 2, 64, 672, 0),          # never: F is no multiple of 128
    ("fp8", 20, 20, 128, 512, 0),       # kv slice of 2560: heads repeated and quantized one after the other
    ("fp8", 4, 1, 64, 768, 65),         # attention; fewer tokens than a sequence, and whole sequences
    ("nvfp4", 8, 2, 64, 1024, 0), ("nvfp4", 4, 2, 80, 768, 65), ("nvfp4", 8, 8, 128, 14336, 0)])
def test_same_bits(b200, mode, n_q, n_kv, hd, ffn, seq_len, tokens):
    if seq_len and tokens > seq_len:
        tokens = tokens // seq_len * seq_len
    stack = _stack(b200, mode, n_q, n_kv, hd, ffn, 2, seq_len, mode == "nvfp4")
    h = torch.randn(tokens, n_q * hd, device="cuda").bfloat16()
    before = h.clone()
    assert stack._native_forward(h) is None     # outside forward() the weights are not promised to be complete
    with b200.capi.gemm_config(static_weights=True):
        assert stack._native_forward(h) is not None
    out = stack.forward(h.view(1, tokens, -1))
    assert out.shape == (1, tokens, n_q * hd) and torch.equal(out[0], _by_calls(stack, h)) and torch.equal(h, before)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = stack.forward(h)
    graph.replay()
    assert torch.equal(captured, out[0]) and b200.capi.device_status() == 0


def test_what_goes_call_by_call(b200):
    capi = b200.capi
    stack = _stack(b200, "nvfp4", 4, 2, 64, 768, 2, 0, False)
    h = torch.randn(32, 256, device="cuda").bfloat16()
    with capi.gemm_config(static_weights=True):
        assert stack._native_forward(h) is None                             # no calibrated ranges
        stack.calibrate(h)
        assert stack._native_forward(h) is not None
        assert stack._native_forward(h.t().contiguous().t()) is None        # not contiguous
        assert stack._native_forward(h.float()) is None
        with capi.gemm_config(tile_n=128):
            assert stack._native_forward(h) is None                         # a forced tile
        stack.layers[1].row_parallel = lambda *a: None
        assert stack._native_forward(h) is None                             # a replaced linear
    stack = _stack(b200, "fp8", 4, 1, 64, 768, 1, 64, False)
    with pytest.raises(ValueError):
        stack.forward(torch.randn(100, 256, device="cuda").bfloat16())      # no whole sequences
    with pytest.raises(ValueError):
        stack.forward(torch.randn(64, 256, device="cuda"))                  # fp32


def _other_backend(stack):
    from tensorrt_b200.stack import CudaBackend
    stack.layers[1].backend = CudaBackend("nvfp4", fuse_gate_up=False)


def _other_config(stack):
    import dataclasses
    stack.layers[0].cfg = dataclasses.replace(stack.cfg, eps=0.5)


REPLACED = {
    "a layer's backend": _other_backend, "a layer's configuration": _other_config,
    **{f"a layer's {n}": (lambda n: lambda stack: setattr(stack.layers[1], n, getattr(stack.layers[1], n)))(n)
       for n in ("forward", "_attention", "_ffn_act", "_amax", "_norm_amax", "_static_amax")},
    **{f"the stack's {n}": (lambda n: lambda stack: setattr(stack, n, getattr(stack, n)))(n) for n in ("_enter", "_walk", "_finish")}}


@pytest.mark.parametrize("what", REPLACED)
def test_replaced_on_an_object(b200, what):
    stack = _stack(b200, "nvfp4", 4, 2, 64, 768, 2, 0, True)
    h = torch.randn(32, 256, device="cuda").bfloat16()
    with b200.capi.gemm_config(static_weights=True):
        assert stack._native_forward(h) is not None
        REPLACED[what](stack)
        assert stack._native_forward(h) is None


@pytest.mark.parametrize("owner,name", [("DecoderStack", "_walk"), ("DecoderLayer", "forward"), ("DecoderLayer", "_amax"), ("CudaBackend", "matmul"),
                                        ("CudaBackend", "add")])
def test_replaced_in_a_class(b200, monkeypatch, owner, name):
    from tensorrt_b200 import stack as module

    stack = _stack(b200, "fp8", 4, 2, 64, 768, 1, 0, False)
    h = torch.randn(32, 256, device="cuda").bfloat16()
    cls = getattr(module, owner)
    orig = getattr(cls, name)
    wrapped = lambda *a, **k: orig(*a, **k)  # noqa: E731
    monkeypatch.setattr(cls, name, staticmethod(wrapped) if name == "add" else wrapped)
    with b200.capi.gemm_config(static_weights=True):
        assert stack._native_forward(h) is None


def test_subclass_of_the_stack(b200):
    from tensorrt_b200.stack import DecoderStack, StackConfig, random_layer_weights

    class Doubled(DecoderStack):
        def _finish(self, h, delta, sharded):
            return super()._finish(h, delta, sharded) * 2

    class Plain(DecoderStack):
        pass

    cfg = StackConfig(hidden=256, n_q=4, n_kv=2, head_dim=64, ffn=768, layers=1)
    h = torch.randn(32, 256, device="cuda").bfloat16()
    out = [cls(cfg, random_layer_weights(cfg, 3)).forward(h) for cls in (DecoderStack, Plain, Doubled)]
    assert torch.equal(out[1], out[0]) and torch.equal(out[2], out[0] * 2)
    with b200.capi.gemm_config(static_weights=True):
        assert Plain(cfg, random_layer_weights(cfg, 3))._native_forward(h) is not None
