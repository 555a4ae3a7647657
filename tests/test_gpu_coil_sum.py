"""Rounding of the coil combine: a product and a sum per coil are rounded once
each, as the error of the whole normal operator at many coils depends on it.

An image of one voxel at the origin, every k-space point sampled, 8 × 8 × 8: the
transforms are exact (equal values, a power of two of them), so that what is
left is the sum over coils, Σ conj(s) (s x).  Its error is at most that of the
same sum formed in FP32 here, by 2 % for the order of a product's two terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def fma(a, b, c):
    return (a.astype(float) * b.astype(float) + c.astype(float)).astype(F)


@pytest.mark.parametrize("Nc", [5, 8])
def test_one_rounding_a_product_and_a_sum(Nc):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(Nc)
    Nt, nvox = 4000, 512
    got, emulated = [], []
    for _ in range(6):
        s = (rng.integers(1, 1 << 11, (Nc, 2)) / 2.0 ** 11).astype(F)      # s x in 21 bits: exact
        x = (rng.integers(1 << 9, 1 << 10, (Nt, 2)) / 2.0 ** 10).astype(F)
        smaps = np.zeros((Nc, 8, 8, 8), np.complex64)
        smaps[:, 0, 0, 0] = s[:, 0] + 1j * s[:, 1]
        img = np.zeros((Nt, 8, 8, 8), np.complex64)
        img[:, 0, 0, 0] = x[:, 0] + 1j * x[:, 1]
        v = (smaps[:, None, 0, 0, 0].astype(complex) * img[None, :, 0, 0, 0].astype(complex)).astype(np.complex64)
        with M.MSLRContext((8, 8, 8), Nc, Nt, nvox, [[8, 8, 8]], [[8, 8, 8]]) as ctx:
            ctx.bind(torch.from_numpy(smaps).cuda(), torch.zeros((Nt, Nc, nvox), dtype=torch.complex64, device="cuda"),
                     torch.arange(nvox, dtype=torch.int32, device="cuda").repeat(Nt, 1))
            out = ctx.normal(torch.from_numpy(img).cuda(), subtract_data=False).cpu().numpy()[:, 0, 0, 0]
        ref = (np.conj(smaps[:, None, 0, 0, 0].astype(complex)) * v).sum(axis=0)
        re, im = np.zeros(Nt, F), np.zeros(Nt, F)
        for c in range(Nc):
            a, b = np.broadcast_to(s[c], (Nt, 2)).T
            re = re + fma(a, v[c].real, b * v[c].imag)
            im = im + fma(a, v[c].imag, -b * v[c].real)
        got.append(out - ref)
        emulated.append(re.astype(float) + 1j * im - ref)
    assert np.linalg.norm(got) <= 1.02 * np.linalg.norm(emulated)
