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


def test_embedding_tokens_are_counted_only_while_that_is_faster():
    """The line between sorting by counting and the library's sort, measured on either side of it."""
    assert 20480 <= _ext.lib().cb_embedding_rank_max() < 24576
