"""The tiled fused step where its tiles, rows and residuals change form, against
the FP64 oracle: loss = Σ(pull(f, ϕ) − g)², df = push(2r), dϕ = Σ_c 2r ∇pull.

Grids at and around the 16 x 8 x 4 tile and every remainder of the x extent modulo
4, mirrored, antisymmetric and circulant boundaries, one to three channels, two
volumes; residuals of image size, of rounding size (g = pull(f, ϕ)) and zero but
for a few voxels; samples outside an ext = 0 band make the loss and their dϕ NaN.

Tolerances: loss 1e-6 relative (a sum of float32 squares); df 4e-6 and dϕ 1e-4 of
the largest element (float32 residuals and derivative weights); with residuals of
rounding size they are themselves rounding, so df is held to push of the residuals
the step must have used, within 1e-6 of the image's scale."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _phi(O, rng, d1, d0, sigma=1.0):
    p = O.identity(d1).astype(np.float64)
    for k in range(3):
        p[..., k] = 1 + (p[..., k] - 1) * (d0[k] - 1) / max(d1[k] - 1, 1)
    return np.asfortranarray((p + sigma * rng.standard_normal(p.shape)).astype(np.float32))


def _step(O, f, phi, g, so):
    r = O.pull(f, phi, so) - g
    gr = O.pull_grad(f, phi, so)
    df = O.push(np.asfortranarray((2 * r).astype(np.float32)), phi, f.shape[:3], so)
    return (r ** 2).sum(), df, (2 * r[:, :, :, None] * gr).sum(axis=4)


@pytest.mark.parametrize("d1", [(16, 8, 4), (17, 9, 5), (15, 7, 6), (34, 18, 9), (35, 40, 33)])
@pytest.mark.parametrize("deg,bnd,nc", [(2, (0, 1, 2), 1), (2, (2, 2, 1), 3), (3, 1, 2), (4, (1, 0, 2), 1)])
def test_tile_edges(pkg, O, d1, deg, bnd, nc):
    L = pkg.layout
    rng = np.random.default_rng(sum(d1) + 10 * deg)
    d0 = (37, 22, 14)
    f = np.asfortranarray(rng.standard_normal(d0 + (nc,)).astype(np.float32))
    g = np.asfortranarray(rng.standard_normal(d1 + (nc,)).astype(np.float32))
    phi = _phi(O, rng, d1, d0)
    loss, df, dphi = pkg.fused_step(L.from_numpy(f), L.from_numpy(phi), L.from_numpy(g), pkg.Settings(deg, bnd, 1))
    rl, rdf, rdp = _step(O, f, phi, g, O.Sett.make(deg, bnd, 1))
    assert abs(float(loss) - rl) <= 1e-6 * rl
    assert rel_err(L.to_numpy(df), rdf) <= 4e-6
    assert rel_err(L.to_numpy(dphi), rdp) <= 1e-4
    assert pkg.native_library().pp_device_status(1) == 0


def test_small_residuals_and_masked_samples(pkg, O):
    L = pkg.layout
    rng = np.random.default_rng(3)
    d = (40, 33, 21)
    f = np.asfortranarray(rng.random(d).astype(np.float32))
    phi = _phi(O, rng, d, d, 0.6)
    s, so = pkg.Settings(2, 1, 1), O.Sett.make(2, 1, 1)
    tf, tp = L.from_numpy(f), L.from_numpy(phi)
    g = pkg.pull(tf, tp, s)
    _, df, _ = pkg.fused_step(tf, tp, g, s)
    assert float(df.abs().max()) <= 1e-6
    few = g.clone()
    few[5, 6, 7] += 1.0
    few[30, 20, 11] -= 2.0
    loss, df, dphi = pkg.fused_step(tf, tp, few, s)
    rl, rdf, rdp = _step(O, f[..., None], phi, L.to_numpy(few)[..., None], so)
    assert abs(float(loss) - rl) <= 1e-6 * rl and rel_err(L.to_numpy(df), rdf[..., 0]) <= 4e-6
    loss, df, dphi = pkg.fused_step(tf, tp, few, pkg.Settings(2, 1, 0))
    ref = O.pull(f, phi, O.Sett.make(2, 1, 0))
    assert np.isnan(ref).any() and np.isnan(float(loss))
    assert np.array_equal(np.isnan(L.to_numpy(dphi)), np.repeat(np.isnan(ref)[..., None], 3, axis=3))
    assert np.isfinite(L.to_numpy(df)).all()
