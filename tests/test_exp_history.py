"""Exp's result has no autograd history (the chain runs on raw device pointers, so a
history could only be a wrong one), whatever its input asks for, and leaves the
input alone.  On the CPU with the native step replaced by a torch one; on the GPU as
it is."""
from __future__ import annotations

import pytest
import torch


def _integer_input(pkg, device):
    v = torch.arange(-6, 18, device=device).reshape(4, 2, 1, 3)
    assert torch.equal(pkg.Exp(v), pkg.Exp(v.float()))
    assert torch.equal(pkg.Exp(v.to(torch.int16)), pkg.Exp(v.float()))
    with pytest.raises(TypeError):
        pkg.Exp(v.double())


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

    def require(*ts):
        if any(t.dtype is not torch.float32 for t in ts):
            raise TypeError("arrays must be Float32")
    monkeypatch.setattr(comp, "_require_cuda", require)

    def step(u, out, last):
        with torch.no_grad():
            out.copy_(u.detach() * 0.5 + float(last))
    monkeypatch.setattr(comp, "_step", step)


@pytest.mark.parametrize("rowmajor", [False, True])
def test_no_history(pkg, torch_steps, rowmajor):
    _check(pkg, _velocity(pkg, "cpu", rowmajor))


def test_integer_velocities(pkg, torch_steps):
    """v / 2^8 of an integer field is float32: such fields are taken as they always were."""
    _integer_input(pkg, "cpu")


@pytest.mark.gpu
def test_integer_velocities_on_the_gpu(pkg):
    _integer_input(pkg, "cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("rowmajor", [False, True])
def test_no_history_on_the_gpu(pkg, rowmajor):
    _check(pkg, _velocity(pkg, "cuda", rowmajor))
