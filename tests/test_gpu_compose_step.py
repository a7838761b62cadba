"""The one-kernel step of Exp (pp_compose_step) against the composition it stands
for, u' = pull(u, id + u), bit by bit: the positions are rounded as the stored
sum and the contraction is the pull kernels' own.  Sizes: one voxel, length-1
axes, a plane that is not a multiple of the block, odd extents; displacements
inside the volume, across the border, several periods out, non-finite."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [(1, 1, 1), (7, 1, 5), (16, 16, 1), (33, 17, 9), (64, 40, 12)])
@pytest.mark.parametrize("amp", [0.03, 2.0, 300.0])
def test_step_matches_compose(pkg, d, amp):
    from pushpull_gb300.compositions import _step, compose
    L = pkg.layout
    rng = np.random.default_rng(int(10 * amp) + sum(d))
    u = (amp * rng.standard_normal(d + (3,))).astype(np.float32)
    if u.size > 30:
        flat = u.reshape(-1)
        flat[[3, 11, 20]] = np.nan, np.inf, 3e9
    u = L.from_numpy(np.asfortranarray(u))
    Id = pkg.id(u)
    ref = compose(u, Id + u)
    out = L.empty(d + (3,))
    _step(u, out, False)
    assert torch.equal(out.nan_to_num(7.0), ref.nan_to_num(7.0)) and torch.equal(out.isnan(), ref.isnan())
    _step(u, out, True)
    ref = ref + Id
    assert torch.equal(out.nan_to_num(7.0), ref.nan_to_num(7.0)) and torch.equal(out.isnan(), ref.isnan())
