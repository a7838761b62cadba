"""pp_fused_step_noalloc on narrow grids, which the fused step takes per voxel: with so
many volumes that the per-voxel kernels' loss partials would not fit the fixed scratch
it runs on the tiled kernels, as it always did, and agrees with pp_fused_step."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [2, 8])
def test_many_narrow_volumes(pkg, nb):
    from pushpull_gb300 import _native as N
    lib, L = pkg.native_library(), pkg.layout
    d, s = (6, 300, 300), pkg.Settings(2, (0, 1, 2), 1)
    gen = torch.Generator().manual_seed(nb)
    col = lambda t: L.colmajor(t.cuda())
    phi = col(pkg.id(dim=d, device="cpu").unsqueeze(-1) + torch.randn(d + (3, nb), generator=gen))
    f, g = (col(torch.rand(d + (1, nb), generator=gen)) for _ in range(2))

    def run(name):
        loss = torch.zeros((), dtype=torch.float64, device="cuda")
        df, dphi = L.empty(tuple(f.shape)), L.empty(tuple(phi.shape))
        rc = getattr(lib, name)(loss.data_ptr(), df.data_ptr(), dphi.data_ptr(), f.data_ptr(), phi.data_ptr(),
                                g.data_ptr(), N.u64x3(d), N.u64x3(d), 1, nb, N.ints(s._packed), 1, N.i32x3(s.deg), 1, 0,
                                torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.pp_last_error()
        return float(loss), df, dphi
    (la, dfa, dpa), (lb, dfb, dpb) = run("pp_fused_step_noalloc"), run("pp_fused_step")
    assert abs(la - lb) <= 1e-6 * lb
    assert float((dfa - dfb).abs().max()) <= 4e-6 * float(dfb.abs().max())
    assert float((dpa - dpb).abs().max()) <= 1e-5 * float(dpb.abs().max())
