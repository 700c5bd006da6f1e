"""What every launch asks of the runtime."""
import types

import pytest
import torch

from chronicals_b200.ops import _ext


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_stream_of_a_torch_without_the_short_way(missing, monkeypatch):
    for name in ("_cuda_getCurrentRawStream", "_cuda_getDevice"):
        monkeypatch.setattr(torch._C, name, lambda *a: 0, raising=False)
    monkeypatch.delattr(torch._C, missing)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=77))
    assert _ext.stream_ptr() == 77
