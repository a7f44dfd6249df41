"""Native whole calls (csrc/python_calls.cpp): `fp8_linear`, `nvfp4_linear`, `fp8_gated_mlp`, `fp8_sdpa`,
`decoder_stack`.  Each returns the result, or None when the call is not the plain case it takes; the caller then goes through `capi`."""
from __future__ import annotations

import importlib.machinery
import importlib.util

from . import _build


def _load():
    _build.build_cuda()
    path = str(_build.build_python_calls())
    loader = importlib.machinery.ExtensionFileLoader("b200q_native", path)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("b200q_native", loader, origin=path))
    loader.exec_module(module)
    return module


_calls = _load()
fp8_linear, nvfp4_linear = _calls.fp8_linear, _calls.nvfp4_linear
fp8_gated_mlp, fp8_sdpa = _calls.fp8_gated_mlp, _calls.fp8_sdpa
decoder_stack = _calls.decoder_stack
