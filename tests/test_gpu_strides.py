"""Strides near 2^31: the second patch is the last one, clamped to the axis's
end, whatever the stride (steps = ⌈(n − p) / s⌉, starts min(i·s, n − p))."""
import numpy as np
import pytest

N, NT, PS = (9, 7, 6), 5, (4, 3, 2)
HUGE = [6, 2**30, 2**31 - 6, 2**31 - 5, 2**31 - 4, 2**31 - 3, 2**31 - 2, 2**31 - 1]


@pytest.mark.parametrize("s", HUGE)
def test_geometry(s):
    from mslr_recon_b200 import recon as R
    ps, steps, Np, starts = R.patch_geometry(N, PS, (s, s, s))
    assert steps == [1, 1, 1] and Np == 8
    assert starts == [[0, n - p] for n, p in zip(N, PS)]
    # long axes: i·s passes 2^31 at the last step
    long = 2**31 - 1
    _, steps, _, starts = R.patch_geometry((long, 1, 1), (7, 1, 1), (2**30, 1, 1))
    assert steps[0] == 2 and starts[0] == [0, 2**30, long - 7]


@pytest.mark.gpu
@pytest.mark.parametrize("s", HUGE)
def test_patches(s):
    import torch
    from mslr_recon_b200 import recon as R
    rng = np.random.default_rng(2)
    img = (rng.standard_normal((NT, 6, 7, 9)) + 1j * rng.standard_normal((NT, 6, 7, 9))).astype(np.complex64)
    d = torch.from_numpy(img).cuda()
    P = R.img2patches(d, PS, (s, s, s))
    where = [(x, y, z) for z in (0, 4) for y in (0, 4) for x in (0, 5)]
    want = np.stack([img[:, z:z + 2, y:y + 3, x:x + 4].reshape(NT, -1) for x, y, z in where])
    assert np.array_equal(P.cpu().numpy().reshape(want.shape), want)
    back = R.patches2img(P, PS, (s, s, s), N).cpu().numpy()   # no two patches meet: copies
    hit = np.zeros(img.shape[1:], bool)
    for x, y, z in where:
        hit[z:z + 2, y:y + 3, x:x + 4] = True
    assert np.array_equal(back, np.where(hit, img, 0))
