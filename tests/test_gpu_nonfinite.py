"""A NaN or an Inf in one patch: that patch comes out non-finite (the reference's
SVD raises an error there), the others as they do without it.  Sides of every
kernel of the split eigen stage, tall and wide patches, in the batched SVST, in
a context's patch SVST and in the nuclear norms."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cn(rng, *s):
    return (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("m,n", [(60, 20), (20, 60), (90, 64), (140, 100), (140, 128), (128, 140), (320, 300), (320, 301)])
def test_one_bad_matrix_of_a_batch(m, n, form, bad):
    import torch
    import mslr_recon_b200 as M
    X = cn(np.random.default_rng(m * n), 5, n, m)
    good = M.svst_batch(dev(X), m, n, [3.0] * 5, form=form)
    for k, (t, l) in {1: (0, 0), 3: (n - 1, m // 2)}.items():
        X[k, t, l] = bad
    out = M.svst_batch(dev(X), m, n, [3.0] * 5, form=form)
    keep = [0, 2, 4]
    assert torch.equal(out[keep], good[keep])
    assert bool(torch.isnan(torch.view_as_real(out[[1, 3]])).all())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_one_bad_voxel_of_a_series(bad):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(5)
    N, Nt = (12, 10, 8), 40
    img = cn(rng, Nt, 8, 10, 12)
    with M.MSLRContext(N, 1, Nt, 1, [[6, 5, 4]], [[6, 5, 4]]) as ctx:
        good, unit = ctx.patch_svst(0, 3.0, dev(img)), ctx.patch_nucnorm(0, dev(img))
        img[17, 2, 7, 9] = bad
        out = ctx.patch_svst(0, 3.0, dev(img))
        assert math.isfinite(unit) and math.isnan(ctx.patch_nucnorm(0, dev(img)))
    hit = torch.zeros(out.shape, dtype=torch.bool, device="cuda")
    hit[:, 0:4, 5:10, 6:12] = True
    assert torch.equal(out[~hit], good[~hit])
    assert bool(torch.isnan(torch.view_as_real(out[hit])).all())
