"""The normal operator with its result over its input: out of a call on X is
what it is with a buffer of its own, bit for bit, for one image series (one
coil group and several; a compiled plane, other lines, and an image without
line kernels) and for a stack of two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 2])
@pytest.mark.parametrize("N,Nc,Nt", [((12, 15, 10), 12, 5), ((12, 15, 10), 12, 400), ((12, 15, 10), 5, 5),
                                     ((32, 32, 24), 13, 26), ((14, 15, 10), 12, 5)])
def test_result_over_the_input(N, Nc, Nt, ns):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(Nc)
    Nx, Ny, Nz = N
    nvox = Nx * Ny * Nz
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()
    idx = np.stack([np.sort(rng.choice(nvox, nvox // 3, replace=False)) for _ in range(Nt)]).astype(np.int32)
    with M.MSLRContext(N, Nc, Nt, nvox // 3, [list(N)], [list(N)]) as ctx:
        ctx.bind(cn(Nc, Nz, Ny, Nx), cn(Nt, Nc, nvox // 3), torch.from_numpy(idx).cuda())
        X = cn(ns, Nt, Nz, Ny, Nx)
        for sub in (True, False):
            want = ctx.normal(X, subtract_data=sub)
            Y = X.clone()
            got = ctx.normal(Y, subtract_data=sub, out=Y[0])
            assert got.data_ptr() == Y.data_ptr() and torch.equal(got, want), sub
