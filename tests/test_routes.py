"""Which kernels a call runs on (pp_get_route; host logic, no GPU): a tile that was set
is used as it is given, the library's own entry chooses by the call."""
from __future__ import annotations

import ctypes as C

import pytest

PULL, GRAD, HESS, PUSH, PUSHG, FUSED, GDOT, HDOT = range(8)
PER_VOXEL, BLOCK, WS, SAMPLED = range(4)


@pytest.fixture
def lib(pkg):
    lib = pkg.native_library()
    yield lib
    assert lib.pp_set_tile(-1, -1, 0, 0, 0, -1) == 0 and lib.pp_set_path(0) == 0


def route(lib, op, deg, d1, d0=None, bnd=(1, 1, 1), nc=1, nb=1, ext=1, ptrs=(256, 256, 256)):
    out = (C.c_int * 5)()
    u = C.c_ulonglong * 3
    rc = lib.pp_get_route(op, *ptrs, u(*(d0 or d1)), u(*d1), nc, nb, C.cast((C.c_int * 3)(*bnd), C.c_void_p), 1,
                          (C.c_int * 3)(*((deg,) * 3 if isinstance(deg, int) else deg)), ext, out)
    assert rc == 0, lib.pp_last_error()
    return tuple(out)


@pytest.mark.parametrize("op", [PULL, GRAD, HESS, GDOT, HDOT])
@pytest.mark.parametrize("deg", [1, 2, 3, 4])
@pytest.mark.parametrize("bnd", [(1, 1, 1), (0, 1, 2)])
@pytest.mark.parametrize("d1", [(40, 36, 44), (41, 35, 43), (192, 192, 39)])
def test_the_warp_specialised_code_is_honoured(lib, op, deg, bnd, d1):
    entry = {GDOT: GRAD, HDOT: HESS}.get(op, op)
    assert lib.pp_set_tile(entry, deg, 3, 3, 4, 15360) == 0
    assert route(lib, op, deg, d1, d0=(96, 96, 97), bnd=bnd) == (WS, 3, 3, 4, 15360)
    assert lib.pp_set_path(1) == 0
    assert route(lib, op, deg, d1, bnd=bnd)[0] == PER_VOXEL


@pytest.mark.parametrize("op,tile", [(PULL, (3, 3, 3, 8192)), (HESS, (4, 3, 2, 6144)), (PUSH, (3, 3, 3, 16384)),
                                     (PUSH, (4, 3, 3, 19968)), (PUSHG, (3, 3, 3, 16384)), (PUSHG, (3, 3, 2, 9984)),
                                     (FUSED, (3, 3, 3, 2560)), (FUSED, (3, 3, 3, 4096))])
@pytest.mark.parametrize("d1", [(40, 36, 44), (192, 192, 192)])
def test_a_set_tile_is_honoured(lib, op, tile, d1):
    for deg in (2, 3, 4):
        assert lib.pp_set_tile(op, deg, *tile) == 0
        assert route(lib, op, deg, d1) == (BLOCK,) + tile
    assert lib.pp_set_tile(op, 3, *tile[:3], 0) == 0
    assert route(lib, op, 3, d1)[0] == PER_VOXEL


def test_back_to_the_own_entry(lib):
    """Read and set again is a choice; cap -1 is the way back."""
    def tile(op, deg):
        v = [C.c_int() for _ in range(4)]
        assert lib.pp_get_tile(op, deg, *[C.byref(x) for x in v]) == 0
        return tuple(x.value for x in v)

    small = (40, 36, 44)
    own = {(op, deg): route(lib, op, deg, small) for op in range(8) for deg in range(5)}
    assert own[PULL, 3][0] == PER_VOXEL and own[FUSED, 2][:4] == (BLOCK, 4, 3, 2)
    seen = {(op, deg): tile(op, deg) for op in range(6) for deg in range(5)}
    for (op, deg), t in seen.items():
        assert lib.pp_set_tile(op, deg, *t) == 0 and tile(op, deg) == t
    assert route(lib, PULL, 3, small)[0] == WS and route(lib, PUSH, 3, small) == (BLOCK, 3, 3, 3, 16384)
    assert lib.pp_set_tile(-1, -1, 0, 0, 0, -1) == 0
    assert {k: route(lib, *k, small) for k in own} == own
    assert {k: tile(*k) for k in seen} == seen


def test_refused(lib):
    for op, t in [(PULL, (4, 3, 3, 8192)), (-1, (4, 3, 3, 8192)), (FUSED, (4, 3, 3, 2560)), (PUSH, (4, 4, 3, 8192)),
                  (PUSH, (3, 3, 4, 8192)), (PULL, (3, 3, 3, -2)), (PULL, (3, 3, 3, 66)), (6, (3, 3, 3, 0))]:
        assert lib.pp_set_tile(op, 3, *t) != 0 and lib.pp_last_error()


@pytest.mark.parametrize("op", [PULL, GRAD, HESS, GDOT, HDOT])
@pytest.mark.parametrize("deg", [2, 3, 4])
@pytest.mark.parametrize("d1", [(192, 192, 39), (192, 192, 96), (192, 60, 192), (60, 192, 192), (192, 60, 100)])
def test_a_slab_goes_where_the_whole_grid_goes(lib, op, deg, d1):
    """A slab of a sample grid spans a part of the image: along that axis the ratio of the
    extents says nothing about the spacing of the samples."""
    d0 = (192, 192, 192)
    assert route(lib, op, deg, d0)[0] == WS
    assert route(lib, op, deg, d1, d0=d0, ptrs=(1 << 34, 256, 1 << 33))[0] == WS


def test_the_deformation_decides_between_a_block_and_a_coarse_grid(lib):
    """n^3 samples over (2n)^3 are every other voxel or a block: by their extents alone
    the same.  Outputs that overlap the deformation leave it to one kernel."""
    far = (1 << 34, 256, 1 << 33)
    for op in (PULL, GRAD, HESS, GDOT, HDOT):
        for deg, n in ((2, 136), (3, 96), (4, 96)):
            d1, d0 = (n, n, n), (2 * n, 2 * n, 2 * n)
            assert route(lib, op, deg, d1, d0=d0, ptrs=far)[0] == SAMPLED
            assert route(lib, op, deg, d1, d0=(n + 20,) * 3, ptrs=far)[0] == WS
            assert route(lib, op, deg, d1, d0=d0, ptrs=(256, 256, 1 << 33))[0] == WS


@pytest.mark.parametrize("op,deg,n,kind,nc,family", [
    (PULL, 2, 64, "clean", 1, PER_VOXEL), (PULL, 2, 80, "clean", 1, WS), (HESS, 3, 80, "clean", 1, WS),
    (GDOT, 3, 72, "clean", 1, PER_VOXEL), (PULL, 4, 64, "clean", 1, PER_VOXEL), (HDOT, 4, 80, "clean", 1, WS),
    (PULL, 1, 160, "clean", 1, PER_VOXEL), (HESS, 1, 128, "clean", 1, WS), (GRAD, 1, 96, "clean", 1, PER_VOXEL),
    (PULL, 2, 128, "circ", 1, WS), (HESS, 3, 128, "circ", 1, WS), (GRAD, 2, 104, "circ", 1, PER_VOXEL),
    (PULL, 4, 96, "circ", 1, WS), (HDOT, 1, 192, "circ", 1, PER_VOXEL),
    (PULL, 2, 181, "odd", 1, PER_VOXEL), (PULL, 3, 97, "odd", 1, PER_VOXEL), (GRAD, 3, 161, "odd", 1, WS),
    (HESS, 4, 97, "odd", 1, PER_VOXEL), (GDOT, 4, 129, "odd", 1, WS), (PULL, 3, 128, "image", 1, WS),
    (HESS, 3, 80, "image", 1, PER_VOXEL), (PULL, 3, 129, "grid", 1, WS), (GRAD, 3, 97, "grid", 1, PER_VOXEL),
    (HESS, 3, 80, "clean", 2, PER_VOXEL), (PULL, 3, 104, "clean", 3, WS), (HDOT, 3, 104, "clean", 3, PER_VOXEL),
    (GDOT, 3, 128, "clean", 3, WS)])
def test_families_by_size_boundary_and_alignment(lib, op, deg, n, kind, nc, family):
    """The families as they measured on both sides of the line (the table in pp_abi.cu):
    clean, circulant margins, rows that are no multiples of 16 bytes in image and grid,
    in the image only, in the grid only."""
    d1 = (n, n, n) if kind in ("clean", "circ", "image") else (n, n + 1, n)
    d0 = {"image": (n + 1, n, n), "grid": (n + 3, n + 1, n)}.get(kind, d1)
    bnd = (1, 0, 1) if kind == "circ" else (1, 1, 2)
    assert route(lib, op, deg, d1, d0=d0, bnd=bnd, nc=nc, ptrs=(1 << 34, 256, 1 << 33))[0] == family


@pytest.mark.parametrize("op", [PULL, GRAD, HESS, GDOT, HDOT])
@pytest.mark.parametrize("deg", [2, 3, 4])
@pytest.mark.parametrize("d1", [(300, 6, 300), (300, 300, 6), (400, 7, 400), (3, 600, 600)])
def test_grids_thinner_than_a_tile(lib, op, deg, d1):
    """Half a tile of the warp-specialised kernels thin: per voxel, and on a tile that was
    set as it was set."""
    assert route(lib, op, deg, d1)[0] == PER_VOXEL
    if d1[0] > 3 and d1[2] > 6:
        assert lib.pp_set_tile({GDOT: GRAD, HDOT: HESS}.get(op, op), deg, 4, 2, 3, 8192) == 0
        assert route(lib, op, deg, d1) == (BLOCK, 4, 2, 3, 8192)


@pytest.mark.parametrize("d1,deg,family", [((6, 300, 300), 2, PER_VOXEL), ((8, 256, 256), 3, PER_VOXEL),
                                           ((4, 256, 256), 4, PER_VOXEL), ((12, 300, 300), 2, PER_VOXEL),
                                           ((12, 300, 300), 3, BLOCK), ((20, 20, 400), 3, BLOCK),
                                           ((300, 6, 300), 3, BLOCK), ((300, 300, 6), 4, BLOCK)])
def test_fused_step_on_narrow_grids(lib, d1, deg, family):
    """Tiles 16 voxels wide on a grid of less than half that: per voxel, unless a tile was set."""
    assert route(lib, FUSED, deg, d1)[0] == family
    if d1[0] > 3:
        assert lib.pp_set_tile(FUSED, deg, 3, 3, 3, 2560) == 0
        assert route(lib, FUSED, deg, d1)[0] == (BLOCK if min(d1) >= 4 else PER_VOXEL)
