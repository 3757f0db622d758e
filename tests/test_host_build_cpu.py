"""Loading of the native host path."""

import pytest
import torch

from velox_voice_b200 import _lib


def test_a_host_module_of_another_build_is_not_loaded(monkeypatch):
    """The module is compiled against one torch, one Python and one C ABI; when it does not belong to the present ones and
    cannot be rebuilt, loading it would call through a wrong layout."""
    _lib.host()  # the present module is there
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(_lib._build, "host_is_current", lambda: False)

    def fails(*a, **k):
        raise RuntimeError("g++ failed")

    monkeypatch.setattr(_lib._build, "build_host", fails)
    with pytest.raises(RuntimeError, match="g\\+\\+ failed"):
        _lib.host()


def test_only_weights_packed_with_natural_scales_are_read_ahead(monkeypatch):
    """GEMM_CONST_B lets a GEMM load its weight under the tail of earlier launches.  A weight that a program assigned without
    natural-layout scales may come from a quantizer that triggers the next launch before it has written."""
    from velox_voice_b200 import _lib, linear, ops

    flags = []

    class Host:
        bsgemm = residual_ln = staticmethod(lambda *a: flags.append(a[-1]) or True)

    monkeypatch.setattr(ops, "_host", lambda: Host)
    layer = linear.PackedLinear.__new__(linear.PackedLinear)
    layer.glu, layer.bias = False, None
    for scales in (torch.zeros(4, 16, dtype=torch.uint8), None):
        layer.q = ops.Quantized(ops.FMT_MX32, 4, 512, torch.zeros(4, 256, dtype=torch.uint8), scales, torch.zeros(1, 4, 512), None)
        layer.forward(layer.q)
        layer.residual_ln(layer.q, residual=None, gamma=None, beta=None, eps=1e-5)
    assert flags == [_lib.GEMM_CONST_B] * 2 + [0] * 2
