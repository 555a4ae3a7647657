"""Equal singular values from parts of a matrix that nothing couples: diagonal
matrices with few distinct values, multiples of the identity, equal blocks, and,
for all eigenpairs, patches with voxels that are exactly zero (coil maps that
end with the object).  Every kernel of the eigen stage, against the FP64 SVST and
the FP64 gradient.

Tolerance: the split-BF16 products' 4·3·2^-17 = 9.2e-5 (FP32 is below that); the
gradient 1e-3 of its scale, as elsewhere."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu

TOL = 9.2e-5


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("n", [3, 8, 9, 25, 32, 50, 64, 96, 128, 130, 301, 400])
def test_equal_singular_values(n, form):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(n)
    m, i = n + 7, np.arange(n)
    few, two, eye = (np.zeros((m, n), complex) for _ in range(3))
    few[rng.permutation(m)[:n], i] = rng.integers(1, 5, n)
    two[i, i] = np.where(i % 2, 1.0, 3.0)
    eye[i, i] = 2.0
    k = max(1, n // 4)
    A = rng.integers(-8, 9, (k, k)) + 1j * rng.integers(-8, 9, (k, k))   # exact products: equal blocks of T
    blocks = np.zeros((m, n), complex)
    for b in range(n // k):
        blocks[b * k:(b + 1) * k, b * k:(b + 1) * k] = A / 8.0
    stack, betas = [few, two, eye, blocks], [0.5, 0.5, 0.5, 0.4]
    cm = torch.from_numpy(np.stack([np.ascontiguousarray(a.T) for a in stack]).astype(np.complex64)).cuda()
    out = M.svst_batch(cm, m, n, betas, form=form).cpu().numpy()
    for q, a in enumerate(stack):
        ref = O.svst(a.astype(np.complex64).astype(complex), betas[q])
        assert np.linalg.norm(out[q].T - ref) <= TOL * np.linalg.norm(a), q


@pytest.mark.parametrize("ps,Nt", [([4, 4, 4], 80), ([2, 2, 2], 20), ([4, 4, 8], 140)])
def test_gradient_with_zero_voxels(ps, Nt):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(Nt)
    N, Nc = (8, 8, 8), 3
    cn = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    smaps = cn(Nc, 8, 8, 8)
    smaps /= np.sqrt((np.abs(smaps) ** 2).sum(0))
    smaps *= rng.random((8, 8, 8)) < 0.6
    smaps = smaps.astype(np.complex64).astype(complex)
    K = 300
    idx = np.sort(rng.random((Nt, 512)).argsort(1)[:, :K], 1).astype(np.int32)
    low = np.einsum("tr,rzyx->tzyx", cn(Nt, 3), cn(3, 8, 8, 8))
    y = (O.sense_forward(low, smaps, idx) + 0.3 * cn(Nt, Nc, K)).astype(np.complex64)
    xt = low.astype(np.complex64)
    prob = O.ReconProblem(smaps=smaps, idx=idx, y=y.astype(complex), patch_sizes=[ps], strides=[ps])
    lam = [0.2 * v for v in prob.lambdas()]
    loss, grad, X, _ = O.pogm_unrolled_grad(prob, 3, xt.astype(complex), lam, 1.0)
    with M.MSLRContext(N, Nc, Nt, K, [ps], [ps]) as ctx:
        ctx.bind(*(torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (smaps.astype(np.complex64), y, idx)))
        ctx.set_lambdas(lam)
        got, g, Xg, _ = ctx.pogm_grad(torch.from_numpy(np.ascontiguousarray(xt)).cuda(), 3, 1.0)
    assert abs(got - loss) <= 1e-3 * loss
    assert np.all(np.abs(np.array(g) - np.array(grad)) <= 1e-3 * np.abs(np.array(grad)).max())
