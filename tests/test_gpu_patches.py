"""Extraction and recombination of patches: starts and covering ranges are
arithmetic on the device, compared here with the enumeration of the starts for
every axis length, patch size and stride up to 11 (clamped, ragged, gapped and
overlapping grids), and on images whose voxels and frames are not multiples of
the kernels' blocks.  Copies are equal; a recombined voxel is a sum of at most
c values and a division in FP32: (c + 1)·2^-24 of their absolute mean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def starts(n, p, s):
    p = min(p, n)
    return p, [min(i * s, n - p) for i in range(-(-(n - p) // s) + 1)]


def check(N, Nt, ps, ss, rng):
    import torch
    from mslr_recon_b200 import recon as R
    ax = [starts(n, p, s) for n, p, s in zip(N, ps, ss)]
    img = (rng.standard_normal((Nt, N[2], N[1], N[0])) + 1j * rng.standard_normal((Nt, N[2], N[1], N[0]))).astype(np.complex64)
    where = [(x, y, z) for z in ax[2][1] for y in ax[1][1] for x in ax[0][1]]
    px, py, pz = (a[0] for a in ax)
    want = np.stack([img[:, z:z + pz, y:y + py, x:x + px].reshape(Nt, -1) for x, y, z in where])
    got = R.img2patches(torch.from_numpy(img).cuda(), ps, ss)
    assert np.array_equal(got.cpu().numpy().reshape(want.shape), want)
    P = (rng.standard_normal(want.shape) + 1j * rng.standard_normal(want.shape)).astype(np.complex64)
    total = np.zeros(img.shape, np.complex128)
    mag = np.zeros(img.shape)
    cnt = np.zeros(img.shape[1:])
    for q, (x, y, z) in zip(P, where):
        box = (slice(None), slice(z, z + pz), slice(y, y + py), slice(x, x + px))
        total[box] += q.reshape(Nt, pz, py, px)
        mag[box] += np.abs(q).reshape(Nt, pz, py, px)
        cnt[box[1:]] += 1
    c = np.maximum(cnt, 1)
    out = R.patches2img(torch.from_numpy(P).cuda(), ps, ss, N).cpu().numpy()
    assert np.all(np.abs(out - total / c) <= (c + 1) * 2.0 ** -24 * mag / c)


def test_every_grid_along_one_axis():
    rng = np.random.default_rng(0)
    for n in range(1, 12):
        for p in range(1, 12):
            for s in range(1, 12):
                axis = (n + p + s) % 3
                N, ps, ss = [1, 1, 1], [1, 1, 1], [1, 1, 1]
                N[axis], ps[axis], ss[axis] = n, p, s
                check(N, 1 + n % 3, ps, ss, rng)


@pytest.mark.parametrize("N,Nt,ps,ss", [((13, 9, 7), 7, (4, 3, 2), (3, 3, 5)), ((17, 16, 2), 8, (7, 7, 2), (2, 3, 1)),
                                        ((10, 11, 12), 17, (10, 11, 12), (4, 4, 4)), ((33, 5, 6), 9, (9, 9, 9), (6, 6, 6))])
def test_ragged_volumes(N, Nt, ps, ss):
    check(N, Nt, ps, ss, np.random.default_rng(1))
