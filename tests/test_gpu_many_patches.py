"""More patches than a dimension of a grid holds: two overlapping scales whose
patches run through one eigen stage, 115 520 in all, and more than 2^31 patches
of one voxel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_overlapping_scales():
    """One iteration against the same iteration with one scale at a time (plain
    form).  Tolerance: split-BF16 Gram, W and rebuild, 4·3·2^-17 = 9.2e-5."""
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(0)
    N, Nc, Nt = (40, 40, 40), 1, 9
    nvox, K = 64000, 20000
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()
    smaps, y = torch.ones((Nc, 40, 40, 40), dtype=torch.complex64, device="cuda"), 10 * cn(Nt, Nc, K)
    idx = torch.from_numpy(np.stack([np.sort(rng.choice(nvox, K, replace=False)) for _ in range(Nt)]).astype(np.int32)).cuda()
    out = {}
    for form in ("plain", "tuned"):
        with M.MSLRContext(N, Nc, Nt, K, [[3, 3, 1], [1, 3, 3]], [[1, 1, 1], [1, 1, 1]], form=form) as ctx:
            ctx.bind(smaps, y, idx)
            ctx.set_lambdas([2.0, 3.0])
            X = ctx.init_x0()
            ctx.pogm_run(X, 1, 2.0)
            out[form] = X
    want = torch.linalg.vector_norm(out["plain"])
    assert float(want) > 0.0
    assert float(torch.linalg.vector_norm(out["tuned"] - out["plain"])) <= 9.2e-5 * float(want)


def test_more_than_2_31_patches():
    import torch
    from mslr_recon_b200 import recon as R
    Nx, Ny, Nz = 2048, 1024, 1025
    img = torch.empty((1, Nz, Ny, Nx), dtype=torch.complex64, device="cuda")
    v = torch.view_as_real(img)
    v[..., 0] = torch.arange(Nx, device="cuda") + 3.0 * torch.arange(Ny, device="cuda")[:, None]
    v[..., 1] = torch.arange(Nz, device="cuda")[:, None, None]
    P = R.img2patches(img, (1, 1, 1), (1, 1, 1))
    assert torch.equal(P.view(-1), img.view(-1))
    del P, img, v
    torch.cuda.empty_cache()   # 34 GB
