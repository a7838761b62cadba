"""The warp-specialised pull's number of CTAs is chosen without a common factor with the
tiles along x: every tile is taken once, at sizes on both sides of the two rounds from
which the choice is made, with tile counts along x that share factors with the full
grid (8, 10, 24) and others; the push of the same grids beside it.

Pull: weights and a 64-term sum in float32, 2e-6 of the largest value.  Push: the
tolerance of a tap's six roundings, at most 27 tiles per element and the fixed-point
words, 2e-6 of the largest value.  A tile left out or taken twice is an error of order
one."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [(64, 160, 128), (64, 144, 128), (80, 144, 144), (79, 145, 143), (192, 96, 96)])
@pytest.mark.parametrize("bnd", [1, (0, 1, 2)])
def test_every_tile_once(pkg, O, d, bnd):
    rng = np.random.default_rng(sum(d))
    L = pkg.layout
    phi = np.asfortranarray((O.identity(d) + 0.7 * rng.standard_normal(d + (3,))).astype(np.float32))
    f = np.asfortranarray((0.2 + rng.random(d)).astype(np.float32))
    s, so = pkg.Settings(3, bnd, 1), O.Sett.make(3, bnd, 1)
    tphi, tf = L.from_numpy(phi), L.from_numpy(f)
    for op, args in (("pull", ()), ("push", (d,))):
        got = L.to_numpy(getattr(pkg, op)(tf, tphi, *args, s))
        ref = getattr(O, op)(f, phi, *args, so)
        e = rel_err(got, ref)
        assert e <= 2e-6, (op, d, e)
    assert pkg.native_library().pp_device_status(1) == 0
