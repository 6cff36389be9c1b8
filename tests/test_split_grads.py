"""Heads of residual blocks of which only one output is used: no work for the other's zeros, and
every parameter still delivers its gradient."""
import importlib

import pytest
import torch

from necklace_b200.ops import LayerNorm, RMSNorm
from necklace_b200.ops.conv import Conv2d
from necklace_b200.parallel.flat import FlatParams

conv_mod = importlib.import_module("necklace_b200.ops.conv")
norm_mod = importlib.import_module("necklace_b200.ops.norm")
DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


def _heads(dev):
    return {"conv": (Conv2d(16, 8, 1, device=dev), (2, 3, 5, 16)),
            "layer_norm": (LayerNorm(16, device=dev), (6, 16)),
            "rms_norm": (RMSNorm(16, device=dev), (6, 16))}


@pytest.mark.parametrize("dev", DEVICES)
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("name", ["conv", "layer_norm", "rms_norm"])
def test_residual_path_alone(dev, flat, name, monkeypatch):
    head, shape = _heads(dev)[name]
    x = torch.randn(shape, device=dev).bfloat16().requires_grad_(True)
    ready = []
    if flat:
        f = FlatParams(head)
        f.grad.fill_(7.0)
        f.set_ready_callback(ready.append)
        f.begin_step()
    alias, _ = head.split(x)

    def unwanted(*a, **k):
        raise AssertionError("a kernel for a gradient of zeros")

    monkeypatch.setattr(conv_mod, "gemm", unwanted)
    monkeypatch.setattr(norm_mod.NormFn, "backward", unwanted)
    d = torch.randn(shape, device=dev).bfloat16()
    alias.backward(d)
    assert torch.equal(x.grad, d)
    for p in head.parameters():
        assert not (p._nkb_grad if flat else p.grad).any()
    assert not flat or len(ready) == len(list(head.parameters()))


@pytest.mark.parametrize("dev", DEVICES)
@pytest.mark.parametrize("name", ["conv", "layer_norm", "rms_norm"])
def test_other_path_alone(dev, name, monkeypatch):
    head, shape = _heads(dev)[name]
    x = torch.randn(shape, device=dev).bfloat16().requires_grad_(True)
    head(x).sum().backward()
    want = [x.grad] + [p.grad for p in head.parameters()]
    x.grad = None
    head.zero_grad()
    seen = []
    gemm, back = conv_mod.gemm, norm_mod.NormFn.backward
    monkeypatch.setattr(conv_mod, "gemm", lambda *a, **k: (seen.append(k.get("res")), gemm(*a, **k))[1])
    monkeypatch.setattr(norm_mod.NormFn, "backward", lambda ctx, dy, dres=None: (
        seen.append(dres), back(ctx, dy, dres))[1])
    head.split(x)[1].sum().backward()
    assert seen and all(s is None for s in seen)
    for a, b in zip(want, [x.grad] + [p.grad for p in head.parameters()]):
        assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -7, atol=1e-2)
