"""The split eigen stage at small Gram sides: its smallest, one and two WY blocks,
a last block of one reflector, and the register tile's edge, against matrices
whose SVST is known in closed form: X = Q₁ diag(s) Q₂ᴴ, SVST = Q₁ diag(max(s −
β, 0)) Q₂ᴴ.

Tolerance: split-BF16 Gram, W and rebuild, 3·2^-17 of a product left out each
and as much for the soft threshold's factor: 4·3·2^-17 = 9.2e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 700])
@pytest.mark.parametrize("n", [8, 9, 15, 16, 17, 18, 24, 31, 32, 33])
def test_small_sides(n, batch):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(1000 * n + batch)
    m = 2 * n + 5
    q1, _ = np.linalg.qr(rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n)))
    q2, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    q1, q2 = torch.from_numpy(q1).cuda(), torch.from_numpy(q2).cuda()
    r = torch.from_numpy(rng.integers(1, n + 1, batch)).cuda()
    i = torch.arange(n, device="cuda")
    s = torch.where(i < r[:, None], 9.0 - 5.0 * i / n, 1.0 - 0.5 * i / n)
    beta = torch.linspace(1.5, 3.0, batch, device="cuda", dtype=torch.float64)
    make = lambda v: (q1 * v[:, None, :].to(q1.dtype)) @ q2.mH
    X = make(s).to(torch.complex64)
    out = M.svst_batch(X.transpose(1, 2).contiguous(), m, n, beta.tolist()).reshape(batch, n, m).transpose(1, 2)
    ref = make((s - beta[:, None]).clamp(min=0.0))
    err = torch.linalg.vector_norm(out - ref, dim=(1, 2)) / torch.linalg.vector_norm(ref, dim=(1, 2))
    assert float(err.max()) <= 9.2e-5
