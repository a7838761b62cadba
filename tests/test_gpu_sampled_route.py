"""Pulls of sample grids that are coarser than the image by their extents run on the
warp-specialised or the per-voxel kernels as a sample of the deformation says.  Exactly
one of the two writes the result: bit by bit the per-voxel kernels' own, whether the
grid spans the image, is a block out of its middle, or mixes both, with masked and
non-finite positions, two volumes and every op.  The output starts as a pattern that
no result has, so that a voxel neither kernel took would show."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _phi(d0, d1, spacing, seed):
    g = torch.Generator().manual_seed(seed)
    p = torch.empty(d1 + (3, 2))
    for k in range(3):
        o = 1.0 + 0.5 * (d0[k] - 1 - spacing * (d1[k] - 1))
        shape = [1, 1, 1, 1]
        shape[k] = -1
        p[..., k, :] = (o + spacing * torch.arange(d1[k], dtype=torch.float32)).view(shape)
    return p + 1.5 * torch.randn(p.shape, generator=g)


@pytest.mark.parametrize("kind", ["coarse", "block", "half", "nan"])
@pytest.mark.parametrize("deg,ext,odd", [(1, 1, 0), (2, 0, 0), (3, 1, 0), (3, 1, 1), (4, 0, 0)])
def test_one_kernel_writes(pkg, kind, deg, ext, odd):
    L, lib = pkg.layout, pkg.native_library()
    d1 = (120 + odd, 112, 96)
    d0 = tuple(2 * n + odd for n in d1)
    phi = _phi(d0, d1, 2.0 if kind == "coarse" else 1.0, deg)
    if kind == "half":
        phi[..., 1] = _phi(d0, d1, 2.0, 7)[..., 1]
    elif kind == "nan":
        phi[torch.rand(phi.shape, generator=torch.Generator().manual_seed(1)) < 0.3] = float("nan")
    phi = L.colmajor(phi.cuda())
    f = L.colmajor(torch.rand(d0 + (2, 2), generator=torch.Generator().manual_seed(2)).cuda())
    up = {"pull_grad_dot": torch.rand(d1 + (2, 2)).cuda(), "pull_hess_dot": torch.rand(d1 + (3, 2, 2)).cuda()}
    s = pkg.Settings(deg, [(1, 0, 2), (2, 1, 1)], bool(ext))
    for op in ("pull", "pull_grad", "pull_hess", "pull_grad_dot", "pull_hess_dot"):
        args = (f, phi, up[op], s) if op in up else (f, phi, s)
        got = getattr(pkg, op)(*args)
        if op not in up:
            out = torch.empty_strided(got.shape, got.stride(), device="cuda").fill_(-7.25e9)
            getattr(pkg, op)(*args, out=out)
            assert torch.equal(out.view(torch.int32), got.view(torch.int32)), op
        assert lib.pp_set_path(1) == 0
        try:
            ref = getattr(pkg, op)(*args)
        finally:
            lib.pp_set_path(0)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.nan_to_num(3.0), ref.nan_to_num(3.0)), op
    assert lib.pp_device_status(1) == 0

