"""W = Ṽ Ṽᴴ of the tuned form: the contraction stops at each patch's rank, and
its operands are split into a BF16 hi and an FP16 lo.  Ranks around the 32-wide
chunks of the contraction and Gram sides around the 128-wide tiles, several
ranks in one batch, against the FP64 SVST.

Tolerance: the Gram and the rebuild carry split-BF16 operands (2^-17 left out
of either factor, lo·lo dropped: at most 3·2^-17 of |M|·|W|), as W's products
do; with the soft threshold's factor of at most one, 4·3·2^-17 = 9.2e-5."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu

TOL = 9.2e-5


@pytest.mark.parametrize("n", [33, 64, 127, 128, 129, 300])
def test_w_stops_at_the_rank(n):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(n)
    m = n + 40
    ranks = sorted({0, 1, 31, 32, min(33, n), min(65, n), n - 1, n})
    stack, betas = [], []
    for r in ranks:
        q1, _ = np.linalg.qr(rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n)))
        q2, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
        s = np.concatenate([np.linspace(9.0, 4.0, r), np.linspace(1.0, 0.5, n - r)])
        stack.append(((q1 * s) @ q2.conj().T).astype(np.complex64))
        betas.append(2.0)
    X = np.stack(stack)
    cm = torch.from_numpy(np.ascontiguousarray(X.transpose(0, 2, 1))).cuda()
    out = np.transpose(M.svst_batch(cm, m, n, betas).cpu().numpy(), (0, 2, 1))
    for k, r in enumerate(ranks):
        ref = O.svst(X[k].astype(np.complex128), betas[k])
        if r == 0:
            assert not np.any(out[k])
        else:
            assert np.linalg.norm(out[k] - ref) / np.linalg.norm(ref) < TOL, r
