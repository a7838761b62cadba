"""The tiled push kernels where their tiles, words and rows end, against the FP64 oracle:

* sample grids at and around the tile sides (16 x 8 x 8, 16 x 8 x 4, 8 x 8 x 4)
  and image extents of every remainder modulo 4, so that the flush meets every
  alignment of a row, planes and channels that start unaligned included;
* values that take each accumulator: image-like (one word), a few values among
  zeros and a large dynamic range (two passes), all zero, noise;
* contracting deformations on both sides of the samples-per-cell threshold,
  with one channel, a full group and a partial group;
* several tiles' worth of samples in one cell.

Tolerance, from the arithmetic: a tap's weight product carries about six float32
roundings (4e-7), an element is added to by at most 27 tiles (27 * 2^-24 / 2 =
8e-7) and the fixed-point words add under 7e-8 of the mean value; relative to the
largest element 2e-6 covers them.  Gradient weights are differences: 4e-6."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = {"push": 2e-6, "push_grad": 4e-6}


def _phi(O, rng, d1, d0, scale=1.0, sigma=0.7):
    p = O.identity(d1).astype(np.float64)
    for k in range(3):
        x = 1 + (p[..., k] - 1) * (d0[k] - 1) / max(d1[k] - 1, 1)
        p[..., k] = 0.5 * (d0[k] + 1) + scale * (x - 0.5 * (d0[k] + 1))
    return np.asfortranarray((p + sigma * rng.standard_normal(p.shape)).astype(np.float32))


def _values(rng, kind, shape):
    if kind == "image":
        v = 0.2 + rng.random(shape)
    elif kind == "sparse":
        v = np.where(rng.random(shape) < 0.01, rng.standard_normal(shape), 0.0)
    elif kind == "range":
        v = rng.standard_normal(shape) * 10.0 ** rng.uniform(-6, 6, shape)
    elif kind == "zero":
        v = np.zeros(shape)
    else:
        v = rng.standard_normal(shape)
    return np.asfortranarray(v.astype(np.float32))


def _check(pkg, O, rng, d0, d1, deg, bnd, ext, nc, kind, scale=1.0, sigma=0.7, phi=None):
    L = pkg.layout
    phi = _phi(O, rng, d1, d0, scale, sigma) if phi is None else phi
    s, so = pkg.Settings(deg, bnd, ext), O.Sett.make(deg, bnd, ext)
    tphi = L.from_numpy(phi)
    for op, extra in (("push", ()), ("push_grad", (3,))):
        f = _values(rng, kind, d1 + extra + (nc,))
        got = L.to_numpy(getattr(pkg, op)(L.from_numpy(f), tphi, d0, s))
        ref = getattr(O, op)(f, phi, d0, so)
        for c in range(nc):
            if not np.abs(ref[..., c]).max() > 0:
                assert not np.any(got[..., c]), (op, c)
                continue
            e = rel_err(got[..., c], ref[..., c])
            assert e <= TOL[op], (op, kind, d0, d1, c, e)
    assert pkg.native_library().pp_device_status(1) == 0


@pytest.mark.parametrize("d1", [(16, 8, 8), (17, 9, 9), (15, 7, 7), (33, 24, 15), (130, 70, 34)])
@pytest.mark.parametrize("d0", [(36, 28, 20), (37, 27, 21), (38, 25, 22), (39, 26, 23)])
def test_tile_and_row_remainders(pkg, O, d0, d1):
    rng = np.random.default_rng(d0[0] * 100 + d1[0])
    _check(pkg, O, rng, d0, d1, 3, (0, 1, 2), 1, 2, "image")


@pytest.mark.parametrize("kind", ["image", "noise", "sparse", "range", "zero"])
@pytest.mark.parametrize("deg", [2, 3, 4])
def test_accumulators(pkg, O, kind, deg):
    rng = np.random.default_rng(deg)
    _check(pkg, O, rng, (41, 36, 30), (41, 36, 30), deg, 1, 1, 1, kind)


@pytest.mark.parametrize("scale", [0.15, 0.3, 0.45, 0.6])
@pytest.mark.parametrize("deg,nc,ext", [(3, 1, 1), (3, 3, 1), (3, 4, 0), (2, 2, 1)])
def test_contraction(pkg, O, scale, deg, nc, ext):
    rng = np.random.default_rng(int(100 * scale) + nc)
    _check(pkg, O, rng, (50, 45, 40), (50, 45, 40), deg, (1, 2, 0), ext, nc, "image", scale, 0.4)


@pytest.mark.parametrize("kind", ["image", "noise"])
def test_all_samples_in_one_cell(pkg, O, kind):
    rng = np.random.default_rng(9)
    d = (32, 16, 16)
    phi = np.empty(d + (3,), np.float32, order="F")
    phi[...] = rng.uniform(9.1, 9.9, d + (3,))
    _check(pkg, O, rng, d, d, 3, 1, 1, 2, kind, phi=phi)
