"""The error text of a checked forward belongs to that call: it comes from the library that ran it and outlives later calls."""
import pytest
import torch

from fused_cpp_b200 import _lib


class _FakeLibrary:
    """Stands for a loaded library whose forward ends with a wait that ran out."""

    def __init__(self, text: bytes):
        self.text = text

    def fmoe_forward_checked(self, *args):
        args[-2]._obj.value, args[-1]._obj.value = _lib.ERR_DEVICE_WAIT, 3
        return _lib.OK

    def fmoe_last_error(self):
        return self.text


@pytest.mark.parametrize("diagnostic", [False, True])
def test_error_text_of_the_call(monkeypatch, diagnostic):
    product, diag = _FakeLibrary(b"from the product library"), _FakeLibrary(b"from the diagnostic library")
    monkeypatch.setattr(_lib, "load", lambda: product)
    monkeypatch.setattr(_lib, "load_diag", lambda: diag)
    monkeypatch.setattr(_lib, "workspace_layout", lambda *shape: _lib.WorkspaceLayout())
    monkeypatch.setattr(_lib, "_require_cuda", lambda name, tensor, dtype: tensor)
    monkeypatch.setattr(_lib, "_stream", lambda: 0)
    x = torch.zeros((2, 16), dtype=torch.bfloat16)
    w13, w2 = torch.zeros((1, 32, 16), dtype=torch.bfloat16), torch.zeros((1, 16, 16), dtype=torch.bfloat16)
    result = _lib.moe_forward(x, w13, w2, torch.ones((2, 1)), torch.zeros((2, 1), dtype=torch.int64), diagnostic=diagnostic, wait=True,
                              workspace=torch.zeros(256, dtype=torch.uint8))
    product.text = diag.text = b"from a later call"
    assert result.status() == (_lib.ERR_DEVICE_WAIT, 3)
    with pytest.raises(_lib.FusedMoEError, match="from the diagnostic library" if diagnostic else "from the product library"):
        result.raise_for_status()
