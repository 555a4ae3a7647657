"""Tensor-core Grams and rebuilds at the edges of their tiles: Gram sides around
the 16 columns an MMA takes, the 64 rows of a half tile and the 128 of a whole
one, contractions around the 16-long chunks (one, two and an odd number of
them), tall and wide, against the FP64 SVST.

Tolerances: three products (Gram, W, rebuild), a fourth share for the soft
threshold's factor of at most one.  Split BF16 leaves 3·2^-17 of a product out:
4·3·2^-17 = 9.2e-5; TF32 rounds both operands by 2^-11: 4·2·2^-11 = 3.9e-3."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [(1, 9.2e-5), (2, 3.9e-3)])
@pytest.mark.parametrize("m,n", [(15, 15), (16, 33), (17, 16), (31, 32), (48, 33), (63, 63), (64, 97), (65, 64), (49, 66),
                                 (113, 127), (130, 128), (129, 145), (150, 130)])
def test_svst_at_tile_edges(m, n, form, tol):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(1000 * m + n)
    k = min(m, n)
    r = (k + 1) // 2
    s = np.concatenate([np.linspace(9.0, 4.0, r), np.linspace(1.0, 0.5, k - r)])
    X, betas = [], [2.0, 2.5, 3.0]
    for _ in betas:
        q1, _ = np.linalg.qr(rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k)))
        q2, _ = np.linalg.qr(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))
        X.append(((q1 * s) @ q2.conj().T).astype(np.complex64))
    cm = torch.from_numpy(np.ascontiguousarray(np.stack(X).transpose(0, 2, 1))).cuda()
    out = np.transpose(M.svst_batch(cm, m, n, betas, form=form).cpu().numpy(), (0, 2, 1))
    for x, o, beta in zip(X, out, betas):
        ref = O.svst(x.astype(np.complex128), beta)
        assert np.linalg.norm(o - ref) <= tol * np.linalg.norm(ref)
