"""The split eigen stage's tridiagonalisation at every kernel edge: the matrix
in registers (tiles of 32, sides 33 to 128) and the blocked form (panels of
16, 64-row chunks, trailing 128; odd and even sides to 384), on matrices with
full and clustered spectra, columns that need no reflection (a diagonal
Gram), rank one and zero, against the FP64 SVST.

Tolerance: Gram, W and rebuild as split-BF16 products, 4·3·2^-17 = 9.2e-5 of
the result (2^-17 left out of either factor, lo·lo dropped)."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu

TOL = 9.2e-5


@pytest.mark.parametrize("n", [33, 34, 49, 50, 63, 65, 95, 96, 97, 126, 130, 131, 143, 144, 145, 160, 191, 193, 256,
                               257, 303, 320, 383, 384])
def test_split_eigen_stage_sides(n):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(n)
    m = n + 17

    def cn(*s):
        return rng.standard_normal(s) + 1j * rng.standard_normal(s)

    q1, _ = np.linalg.qr(cn(m, n))
    q2, _ = np.linalg.qr(cn(n, n))
    diag = np.zeros((m, n), complex)
    diag[np.arange(n), np.arange(n)] = np.linspace(7, 3, n)
    stack = [cn(m, n), (q1 * np.repeat([9.0, 5.0, 1.0], -(-n // 3))[:n]) @ q2.conj().T, diag,
             np.outer(cn(m), cn(n)), np.zeros((m, n), complex), q1 * np.linspace(6, 2, n)]
    betas = [2.0, 2.0, 4.0, 1.0, 1.0, 3.0]
    X = np.stack([a.astype(np.complex64) for a in stack])
    cm = torch.from_numpy(np.ascontiguousarray(X.transpose(0, 2, 1))).cuda()
    out = np.transpose(M.svst_batch(cm, m, n, betas).cpu().numpy(), (0, 2, 1))
    for k in range(len(stack)):
        ref = O.svst(X[k].astype(np.complex128), betas[k])
        nr = np.linalg.norm(ref)
        assert np.linalg.norm(out[k] - ref) <= TOL * nr, (k, np.linalg.norm(out[k] - ref) / max(nr, 1e-30))
