"""A GEMM behind a quantize kernel that was asked to let its dependents go late may request its weight tiles at once, whatever wrote
them (common.cuh::pdl_enter).  So no way through such a quantizer may launch a kernel that does not know of `late`."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "tensorrt_b200" / "csrc"
# what stands in front of the quantize kernel itself (the abs-max, clearing a scale tile), and a cast of the stream
IN_FRONT = {"b200q_amax", "cudaMemsetAsync", "static_cast"}


def _closing(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def _launches_without_late(text):
    text = re.sub(r"//[^\n]*", "", text)
    bad = []
    for f in re.finditer(r"\bint (\w+)\(([^)]*\bbool late\b[^)]*)\)\s*\{", text):
        body = text[f.end() - 1:_closing(text, f.end() - 1, "{}")]
        for call in re.finditer(r"\b(\w+)(?:<[^<>()]*(?:<[^<>()]*>)?[^<>()]*>)?\(", body):
            args = body[call.end():_closing(body, call.end() - 1, "()")]
            on_stream = re.search(r"(^|,)\s*(st|stream|&cfg)\s*(,|$)", args)
            if on_stream and call[1] not in IN_FRONT and not re.search(r"\blate\b", args):
                bad.append((f[1], call[1]))
    return bad


def test_every_launch_of_a_late_quantizer_is_told():
    seen = ""
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        seen += text
        assert _launches_without_late(text) == [], path.name
    assert "int launch_fp8_rows_stream(" in seen and "int silu_mul_fp8_quantize(" in seen
    assert _launches_without_late("int f(cudaStream_t st, bool late) {\n  return g<T, 1>(x, st);\n}") == [("f", "g")]


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n,k", [(1200, 1024, 28672), (1184, 1536, 16512)])
def test_weights_written_directly_in_front(b200, rows, n, k):
    """Rows that the streaming quantizer takes, in front of a GEMM over blocks of tokens: the module called behind its own
    constructor against the same call on weights that are long complete."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    for _ in range(4):
        w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).bfloat16()
        torch.cuda.synchronize()
        module = b200.linear.Fp8Linear.from_float(w)
        at_once = module(x)
        torch.cuda.synchronize()
        assert torch.equal(at_once, module(x))
    assert b200.capi.device_status() == 0
