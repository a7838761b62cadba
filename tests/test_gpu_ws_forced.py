"""The warp-specialised pull kernels on every way they load a tile, at sizes where the
library itself would go per voxel: the tile is set, pp_get_route has to say that it is
taken, and every op gives the bits of the per-voxel kernels.

* image and sample rows of every remainder modulo four floats: boxes by TMA, by TMA from
  a row-padded copy, deformations by TMA or copied by the threads that read them;
* mirrored, circulant and mixed margins, several channels with boundaries of their own,
  two volumes, masked samples;
* an image whose padded copy is not made, because it is over four times the grid or the
  stream is being captured: boxes loaded row by row one unit ahead, under both ways of
  the deformation;
* more tiles than CTAs, several rounds of them, at tile counts with and without a
  common factor."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

OPS = {"pull": 0, "pull_grad": 1, "pull_hess": 2, "pull_grad_dot": 6, "pull_hess_dot": 7}


@pytest.fixture
def lib(pkg):
    lib = pkg.native_library()
    for op in (0, 1, 2):
        assert lib.pp_set_tile(op, -1, 3, 3, 4, 15360) == 0
    yield lib
    assert lib.pp_set_tile(-1, -1, 0, 0, 0, -1) == 0 and lib.pp_set_path(0) == 0


def _inputs(pkg, d0, d1, nc, nb, spacing=None, sigma=1.2, seed=0):
    L, g = pkg.layout, torch.Generator().manual_seed(seed)
    phi = torch.empty(d1 + (3, nb))
    for k in range(3):
        h = spacing or (d0[k] - 1) / max(d1[k] - 1, 1)
        shape = [1, 1, 1, 1]
        shape[k] = -1
        phi[..., k, :] = (0.5 * (d0[k] + 1) + h * (torch.arange(d1[k]) - 0.5 * (d1[k] - 1))).view(shape)
    phi += sigma * torch.randn(phi.shape, generator=g)
    f = torch.randn(d0 + (nc, nb), generator=g)
    up = {"pull_grad_dot": torch.randn(d1 + (nc, nb), generator=g),
          "pull_hess_dot": torch.randn(d1 + (3, nc, nb), generator=g)}
    col = lambda t: L.colmajor(t.cuda())
    return col(f), col(phi), {k: col(v) for k, v in up.items()}


def _route(lib, op, f, phi, s):
    route, n = (C.c_int * 5)(), C.c_ulonglong * 3
    rc = lib.pp_get_route(OPS[op], 256, phi.data_ptr(), f.data_ptr(), n(*f.shape[:3]), n(*phi.shape[:3]), f.shape[3],
                          f.shape[4], s.bnd_array(), s.nbnd, (C.c_int * 3)(*s.deg), s.ext, route)
    assert rc == 0, lib.pp_last_error()
    return tuple(route)


def _same(a, b):
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(3.0), b.nan_to_num(3.0))


def _against_per_voxel(pkg, lib, f, phi, up, s, ops=tuple(OPS)):
    got = {}
    for op in ops:
        args = (f, phi, up[op], s) if op in up else (f, phi, s)
        assert _route(lib, op, f, phi, s)[0] == 2
        got[op] = getattr(pkg, op)(*args)
        assert lib.pp_set_path(1) == 0
        try:
            ref = getattr(pkg, op)(*args)
        finally:
            lib.pp_set_path(0)
        assert _same(got[op], ref), op
    assert lib.pp_device_status(1) == 0
    return got


@pytest.mark.parametrize("x0", [40, 41, 42, 43])
@pytest.mark.parametrize("x1", [40, 41, 42, 43])
@pytest.mark.parametrize("bnd", [1, 2, 0, (0, 1, 2)])
def test_rows_modulo_four(pkg, O, lib, x0, x1, bnd):
    f, phi, up = _inputs(pkg, (x0, 30, 29), (x1, 37, 33), 2, 1, seed=x0 * 64 + x1)
    s = pkg.Settings(3, bnd, 1)
    got = _against_per_voxel(pkg, lib, f, phi, up, s)
    if x0 == x1:
        L = pkg.layout
        ref = O.pull(L.to_numpy(f), L.to_numpy(phi), O.Sett.make(3, bnd, 1))
        assert rel_err(L.to_numpy(got["pull"]), ref) <= 1e-5


@pytest.mark.parametrize("deg", [1, 2, 3, 4])
@pytest.mark.parametrize("x0,x1", [(48, 48), (47, 48), (48, 45), (45, 47)])
@pytest.mark.parametrize("ext", [0, 1])
def test_degrees_channels_volumes(pkg, lib, deg, x0, x1, ext):
    f, phi, up = _inputs(pkg, (x0, 35, 31), (x1, 33, 46), 3, 2, seed=deg)
    _against_per_voxel(pkg, lib, f, phi, up, pkg.Settings(deg, [(1, 2, 0), (0, 0, 1), (2, 1, 1)], ext))


@pytest.mark.parametrize("deg", [1, 2, 3, 4])
@pytest.mark.parametrize("x1", [40, 41])
@pytest.mark.parametrize("nc", [1, 3])
def test_image_over_four_times_the_grid(pkg, lib, deg, x1, nc):
    """No copy: every box row by row, one unit ahead; blocks of spacing one out of the image's
    middle and, for tiles at the border and beyond a buffer, the whole of it."""
    for spacing in (1.0, None):
        f, phi, up = _inputs(pkg, (91, 82, 83), (x1, 50, 49), nc, 2, spacing=spacing, seed=deg + nc)
        _against_per_voxel(pkg, lib, f, phi, up, pkg.Settings(deg, (0, 1, 2), 1))


@pytest.mark.parametrize("x0,x1", [(48, 48), (47, 48), (47, 45), (48, 45)])
@pytest.mark.parametrize("nc", [1, 2])
def test_capture(pkg, lib, x0, x1, nc):
    """While a stream is captured no scratch is allocated: unaligned images are read where
    they are.  Replays on new values in the same arrays."""
    f, phi, up = _inputs(pkg, (x0, 44, 40), (x1, 48, 46), nc, 2, seed=nc)
    s = pkg.Settings(3, (2, 1, 0), 1)
    ops = ("pull", "pull_grad", "pull_hess")
    outs = [torch.empty_strided(r.shape, r.stride(), device="cuda")
            for r in (getattr(pkg, op)(f, phi, s) for op in ops)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for op, out in zip(ops, outs):
            getattr(pkg, op)(f, phi, s, out=out)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for op, out in zip(ops, outs):
            getattr(pkg, op)(f, phi, s, out=out)
    for seed in (11, 12):
        f2, phi2, _ = _inputs(pkg, (x0, 44, 40), (x1, 48, 46), nc, 2, seed=seed)
        f.copy_(f2)
        phi.copy_(phi2)
        graph.replay()
        assert lib.pp_set_path(1) == 0
        try:
            refs = [getattr(pkg, op)(f, phi, s) for op in ops]
        finally:
            lib.pp_set_path(0)
        assert all(_same(a, b) for a, b in zip(outs, refs))
    assert lib.pp_device_status(1) == 0


@pytest.mark.parametrize("d", [(64, 160, 128), (79, 145, 143), (192, 96, 96), (81, 100, 135)])
@pytest.mark.parametrize("bnd", [1, (0, 1, 2)])
def test_every_tile_once(pkg, lib, d, bnd):
    f, phi, up = _inputs(pkg, d, d, 1, 1, sigma=0.7, seed=sum(d))
    _against_per_voxel(pkg, lib, f, phi, up, pkg.Settings(3, bnd, 1), ("pull", "pull_grad", "pull_grad_dot"))


def test_unaligned_base(pkg, lib):
    """Arrays that start 4 bytes past a 16-byte address."""
    f, phi, up = _inputs(pkg, (48, 40, 36), (48, 36, 45), 2, 1)
    L, s = pkg.layout, pkg.Settings(3, (1, 0, 2), 1)

    def shift(t):
        store = torch.empty(t.numel() + 1, device="cuda")
        v = L.unflat(store[1:], tuple(t.shape))
        v.copy_(t)
        return v
    ref = _against_per_voxel(pkg, lib, f, phi, up, s)
    for fs, ps in ((shift(f), phi), (f, shift(phi)), (shift(f), shift(phi))):
        got = _against_per_voxel(pkg, lib, fs, ps, up, s)
        assert all(_same(got[k], ref[k]) for k in ref)
