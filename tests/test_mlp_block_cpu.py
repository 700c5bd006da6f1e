"""The gated MLP calls whatever stands in for its down projection."""
import pytest
import torch

from chronicals_b200 import ChronicalsConfig, ops
from chronicals_b200.models.decoder import MLP, FusedLinear


def _mlp():
    torch.manual_seed(0)
    m = MLP(ChronicalsConfig.from_model_name("tiny-qwen2"), torch.float32)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    return m


class _Other(torch.nn.Module):
    """Any module that takes ``(x, residual)``."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x, residual):
        return 2 * self.inner(x) + residual


class _Scaled(FusedLinear):
    def forward(self, x, residual=None):
        return 2 * super().forward(x) + residual


def _replace(m):
    m.down_proj = _Other(m.down_proj)


def _subclass(m):
    m.down_proj.__class__ = _Scaled


def _patch(m):
    plain = m.down_proj.forward
    m.down_proj.forward = lambda x, residual=None: 2 * plain(x) + residual


def _hook(m):
    m.down_proj.register_forward_hook(lambda mod, args, out: 2 * out - args[1])


def _global_hook(m):
    def twice(mod, args, out):
        return 2 * out - args[1] if mod is m.down_proj else None
    return torch.nn.modules.module.register_module_forward_hook(twice)


@pytest.mark.parametrize("change", [_replace, _subclass, _patch, _hook, _global_hook])
def test_a_changed_down_projection_is_called(change):
    m = _mlp()
    x, r = torch.randn(5, m.gate_up_proj.in_features), torch.randn(5, m.gate_up_proj.in_features)
    plain = m(x, r)
    handle = change(m)
    try:
        got = m(x, r)
    finally:
        if handle is not None:
            handle.remove()
    assert torch.allclose(got, 2 * (plain - r) + r, atol=1e-5)


def test_an_unchanged_one_is_part_of_the_block(monkeypatch):
    m, calls = _mlp(), []
    block = ops.swiglu_mlp
    monkeypatch.setattr(ops, "swiglu_mlp", lambda *a: calls.append(1) or block(*a))
    x = torch.randn(3, m.gate_up_proj.in_features)
    m(x, torch.zeros_like(x))
    assert calls
