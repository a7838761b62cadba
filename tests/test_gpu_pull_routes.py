"""The pull family's routes by size, degree and alignment give the same bits.

The per-voxel kernels, the warp-specialised kernels and their ways of loading a
box (TMA window, mirrored margins, rows loaded by the threads, a row-padded copy
of the image) share one contraction, so that a grid computed whole and the same
grid computed in parts, which may take other kernels, agree exactly.  Each case
compares the default route with the per-voxel one bit by bit and with the FP64
oracle (norm-wise 1e-5 for pull, 1e-4 for the derivatives):

* image and sample extents of every remainder modulo 4 (TMA cannot address odd ones);
* mirrored, circulant and mixed boundaries, with and without extrapolation;
* sizes on both sides of the rule that picks the kernels;
* an image much larger than the sample grid (no padded copy), a base address
  that is not 16-byte aligned, and a stream under graph capture."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _phi(O, rng, d1, d0, sigma=1.5):
    p = O.identity(d1).astype(np.float64)
    for k in range(3):
        p[..., k] = 1 + (p[..., k] - 1) * (d0[k] - 1) / max(d1[k] - 1, 1)
    return np.asfortranarray((p + sigma * rng.standard_normal(p.shape)).astype(np.float32))


def _compare(pkg, O, d0, d1, deg, bnd, ext, nc=1, oracle=True):
    lib, L = pkg.native_library(), pkg.layout
    rng = np.random.default_rng(sum(d0) + sum(d1) + deg)
    f0 = np.asfortranarray(rng.standard_normal(d0 + (nc,)).astype(np.float32))
    phi = _phi(O, rng, d1, d0)
    s, so = pkg.Settings(deg, bnd, ext), O.Sett.make(deg, bnd, ext)
    tf, tp = L.from_numpy(f0), L.from_numpy(phi)
    for op, tol in (("pull", 1e-5), ("pull_grad", 1e-4)):
        got = L.to_numpy(getattr(pkg, op)(tf, tp, s))
        assert lib.pp_set_path(1) == 0
        try:
            direct = L.to_numpy(getattr(pkg, op)(tf, tp, s))
        finally:
            lib.pp_set_path(0)
        assert np.array_equal(got, direct, equal_nan=True), (op, d0, d1)
        if oracle:
            assert rel_err(got, getattr(O, op)(f0, phi, so)) <= tol, (op, d0, d1)
    assert lib.pp_device_status(1) == 0


@pytest.mark.parametrize("x0", [72, 73, 74, 75])
@pytest.mark.parametrize("x1", [72, 73, 74, 75])
@pytest.mark.parametrize("bnd", [1, 2, 0, (0, 1, 2)])
def test_extents_modulo_four(pkg, O, x0, x1, bnd):
    _compare(pkg, O, (x0, 50, 49), (x1, 92, 91), 3, bnd, 1, nc=2, oracle=x0 == x1)


@pytest.mark.parametrize("deg", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("d1", [(40, 40, 40), (100, 92, 92), (101, 92, 92), (132, 128, 130)])
def test_sizes_around_the_rule(pkg, O, deg, d1):
    _compare(pkg, O, (64, 60, 56), d1, deg, 1, 0, oracle=d1[0] <= 101)


def test_padded_copy_limits(pkg, O):
    _compare(pkg, O, (181, 150, 140), (84, 80, 84), 4, 1, 1)          # image much larger than the grid


def test_unaligned_base_and_capture(pkg, O):
    L = pkg.layout
    rng = np.random.default_rng(4)
    d0, d1 = (72, 70, 68), (120, 92, 92)
    f0 = np.asfortranarray(rng.standard_normal(d0).astype(np.float32))
    phi = _phi(O, rng, d1, d0)
    s = pkg.Settings(3, 1, 1)
    tp = L.from_numpy(phi)
    ref = pkg.pull(L.from_numpy(f0), tp, s)
    store = torch.empty(f0.size + 1, device="cuda")
    odd = L.unflat(store[1:], d0)                                       # 4 bytes past an aligned address
    odd.copy_(L.from_numpy(f0))
    assert torch.equal(pkg.pull(odd, tp, s), ref)
    out = L.empty(d1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        pkg.pull(odd, tp, s, out=out)
    torch.cuda.current_stream().wait_stream(side)
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.pull(odd, tp, s, out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
