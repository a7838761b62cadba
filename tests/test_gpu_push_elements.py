"""Push, push_grad, the affine push and the fused step's image gradient element by
element: where bright and dark values share a tile, where the sample grid ends, and
under contraction, against 64 bits.

Bound on an element's error.  S: the sum of the absolute values of its contributions.
A contribution is a product of weights and a value in float32, about seven roundings,
and reaches the image through at most 27 tiles' sums, each rounded once and added in
float32: 34 * 2^-24 S = 2.0e-6 S.  (Gradients: three products and their sum, derivative
weights from differences: twice that.)  In a tile contributions are summed in fixed point
with a quantum of at most 2^(E - 43).  Per voxel: 2^E <= 4 max|v| (max|v| < 2^E / 2 or
the tile's sum of up to 512 values < 2^(E + 7)), half a quantum each, one contribution
per voxel: 512 * 2^-42 max|v| = 1.2e-10 max|v| from one tile; an element near that small
has contributions from few voxels, but all are allowed here.  A contracted tile's
voxels are summed in float32, 16 at a time in either half (8 * 2^-24 S more at most),
with a quantum 2^-43 of twice the tile's sum, 512 * 2 * 2^-44 max|v| a rounding, one per
cell and run of 32 voxels: at most 64 + 16 of them, 5e-9 max|v|.  push_grad's values
count with their three components' sum and a factor of two."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bspline(t, n):
    if n < 0:
        return np.zeros_like(t)
    if n == 0:
        return ((t > -0.5) & (t <= 0.5)).astype(np.float64)
    h = 0.5 * (n + 1)
    return ((h + t) * _bspline(t + 0.5, n - 1) + (h - t) * _bspline(t - 0.5, n - 1)) / n


def _push64(phi, v, d0, deg):
    """(push or push_grad of v, the sum of the contributions' absolute values), reflecting
    boundary, in 64 bits from the float32 positions."""
    x = (phi.reshape(-1, 3, order="F") - np.float32(1.0)).astype(np.float32)
    o = np.ceil(x - np.float32(0.5 * (deg + 1))).astype(np.int64)
    axes = []
    for k in range(3):
        taps = []
        for i in range(deg + 1):
            t = x[:, k].astype(np.float64) - (o[:, k] + i)
            r = (o[:, k] + i) % (2 * d0[k])
            dw = _bspline(t + 0.5, deg - 1) - _bspline(t - 0.5, deg - 1)
            taps.append((np.where(r >= d0[k], 2 * d0[k] - 1 - r, r), _bspline(t, deg), dw))
        axes.append(taps)
    n0 = d0[0] * d0[1] * d0[2]
    out, S = np.zeros(n0), np.zeros(n0)
    grad = v.ndim == 4
    g = v.reshape((-1, 3) if grad else (-1, 1), order="F").astype(np.float64)
    for iz, wz, dz in axes[2]:
        for iy, wy, dy in axes[1]:
            for ix, wx, dx in axes[0]:
                at = ix + d0[0] * (iy + d0[1] * iz)
                parts = ((dx * wy * wz, wx * dy * wz, wx * wy * dz) if grad else (wx * wy * wz,))
                terms = [w * g[:, p] for p, w in enumerate(parts)]
                out += np.bincount(at, sum(terms), n0)
                S += np.bincount(at, sum(np.abs(t) for t in terms), n0)
    return out.reshape(d0, order="F"), S.reshape(d0, order="F")


def _phi(rng, d1, d0, scale):
    p = np.empty(d1 + (3,))
    for k in range(3):
        x = 0.5 * (d0[k] - 1) + scale * (np.arange(d1[k]) - 0.5 * (d1[k] - 1))
        p[..., k] = 1 + x.reshape([-1 if k == a else 1 for a in range(3)])
    return np.asfortranarray((p + 0.3 * rng.standard_normal(p.shape)).astype(np.float32))


def _stripes(rng, d1, kind, tail=()):
    """Values in 0.5 .. 1.5; every other 8 planes along an axis of the tile 1e-4 as large,
    or one voxel in 64 as it is and the others 1e-5 as large."""
    v = (0.5 + rng.random(d1 + tail)) * np.where(rng.random(d1 + tail) < 0.5, -1, 1) ** (len(tail) > 0)
    if kind == "few":
        m = rng.random(d1) < 1 / 64
        v *= np.where(m, 1.0, 1e-5).reshape(d1 + (1,) * len(tail))
    else:
        k = "xyz".index(kind)
        m = np.where((np.arange(d1[k]) // 4) % 2 == 0, 1.0, 1e-4)
        v *= m.reshape([-1 if k == a else 1 for a in range(3)] + [1] * len(tail))
    return np.asfortranarray(v.astype(np.float32))


def _check(got, out, S, vmax, rel, dense):
    tol = rel * S + (5e-9 if dense else 1.2e-10) * vmax
    bad = np.abs(got.astype(np.float64) - out) > tol
    assert not bad.any(), (int(bad.sum()), float((np.abs(got - out) / tol).max()))


@pytest.mark.parametrize("kind", ["x", "y", "z", "few"])
@pytest.mark.parametrize("deg,scale", [(2, 1.0), (3, 1.0), (4, 1.0), (2, 0.3), (3, 0.45), (3, 0.25), (4, 0.25), (3, 0.1)])
def test_push_and_push_grad(pkg, kind, deg, scale):
    L = pkg.layout
    rng = np.random.default_rng(deg * 10 + "xyzfew".index(kind[0]))
    d1 = d0 = (56, 44, 42)
    phi = _phi(rng, d1, d0, scale)
    tphi, s = L.from_numpy(phi), pkg.Settings(deg, 1, 1)
    dense = scale <= 0.45
    v = _stripes(rng, d1, kind)
    _check(L.to_numpy(pkg.push(L.from_numpy(v), tphi, d0, s)), *_push64(phi, v, d0, deg), 1.5, 2e-6, dense)
    g = _stripes(rng, d1, kind, (3,))
    _check(L.to_numpy(pkg.push_grad(L.from_numpy(g), tphi, d0, s)), *_push64(phi, g, d0, deg), 2 * 4.5, 4e-6, dense)
    assert pkg.native_library().pp_device_status(1) == 0


@pytest.mark.parametrize("kind", ["x", "few"])
@pytest.mark.parametrize("deg", [2, 3, 4])
def test_fused_and_affine(pkg, kind, deg):
    """The fused step of an image of zeros pushes -2 g; the affine push of the grid's own
    positions, at a fraction of a voxel, is a push."""
    L = pkg.layout
    rng = np.random.default_rng(100 + deg)
    d = (56, 44, 42)
    s = pkg.Settings(deg, 1, 1)
    v = _stripes(rng, d, kind)
    phi = _phi(rng, d, d, 1.0)
    _, df, _ = pkg.fused_step(L.zeros(d), L.from_numpy(phi), L.from_numpy(v), s)
    out, S = _push64(phi, v, d, deg)
    _check(L.to_numpy(df), -2 * out, 2 * S, 3.0, 2e-6, False)
    A = np.eye(4, dtype=np.float32)
    A[:3, 3] = 0.25, -0.375, 0.5
    got = L.to_numpy(pkg.affine_push(L.from_numpy(v), A, d, s))
    phi = np.empty(d + (3,), np.float32, order="F")
    for k in range(3):
        phi[..., k] = (1 + np.arange(d[k], dtype=np.float32) + A[k, 3]).reshape([-1 if k == a else 1 for a in range(3)])
    _check(got, *_push64(phi, v, d, deg), 1.5, 2e-6, False)
