"""Exp's result has no autograd history (the chain runs on raw device pointers, so a
history could only be a wrong one), whatever its input asks for, and leaves the
input alone.  On the CPU with the native step replaced by a torch one; on the GPU as
it is."""
from __future__ import annotations

import pytest
import torch


def _velocity(pkg, device, rowmajor):
    g = torch.Generator().manual_seed(5)
    v = torch.rand((6, 5, 4, 3), generator=g) - 0.5
    v = v.to(device) if rowmajor else pkg.layout.colmajor(v.to(device))
    return v.requires_grad_(True)


def _check(pkg, v):
    before = v.detach().clone()
    out = pkg.Exp(v)
    assert not out.requires_grad and out.grad_fn is None
    with pytest.raises(RuntimeError):
        out.sum().backward()
    assert v.grad is None and torch.equal(v.detach(), before)
    assert torch.equal(out, pkg.Exp(before))


@pytest.fixture
def torch_steps(pkg, monkeypatch):
    """The native step's contract on CPU tensors: writes ``out`` behind autograd's back."""
    import pushpull_gb300.compositions as comp
    monkeypatch.setattr(comp, "_require_cuda", lambda *ts: None)

    def step(u, out, last):
        with torch.no_grad():
            out.copy_(u.detach() * 0.5 + float(last))
    monkeypatch.setattr(comp, "_step", step)


@pytest.mark.parametrize("rowmajor", [False, True])
def test_no_history(pkg, torch_steps, rowmajor):
    _check(pkg, _velocity(pkg, "cpu", rowmajor))


@pytest.mark.gpu
@pytest.mark.parametrize("rowmajor", [False, True])
def test_no_history_on_the_gpu(pkg, rowmajor):
    _check(pkg, _velocity(pkg, "cuda", rowmajor))
