"""Scratch that the library takes outside the caller's allocator: a pull of an image that
needs a padded copy leaves at most 64 MiB taken once it is done, and nothing after
pp_release_scratch; results before and after are the same."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def test_kept_and_given_back(pkg):
    L, lib = pkg.layout, pkg.native_library()
    d, nc = (257, 251, 253), 3                                    # a copy of 190 MiB
    phi = pkg.id(dim=d)
    phi += 0.3
    f = L.colmajor(torch.rand(d + (nc,), device="cuda"))
    out, first, s = L.empty(d + (nc,)), L.empty(d + (nc,)), pkg.Settings(3, 1, True)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    pkg.pull(f, phi, s, out=first)                                # the kernels are loaded from here on
    out.zero_()
    assert not torch.equal(first, out)                            # (what torch takes for it, it has)
    assert lib.pp_release_scratch() == 0
    nothing = free()
    pkg.pull(f, phi, s, out=out)
    kept = nothing - free()
    assert torch.equal(out, first)
    assert lib.pp_release_scratch() == 0
    assert free() == nothing
    assert 0 <= kept <= 64 * MIB, kept / MIB
    out.zero_()
    pkg.pull(f, phi, s, out=out)
    assert torch.equal(out, first)
