"""FP32 tiles of the CUDA cores: the plain form's Gram and rebuild and the
gradient's products, at sides around the 64-wide tiles and contractions around
the 16-long slices, tall and wide, against FP64.

Tolerances.  SVST: sums of at most 200 FP32 terms carry 200·2^-24 = 1.2e-5 of
the operands' norms in the Gram, and as much again in the rebuild of a matrix
whose kept singular values are well apart from the threshold: 2.4e-5.
Gradient: five iterations, each contributing the iterate's 1e-4 twice (the
adjoint and the iterate it is multiplied with): 1e-3 of the largest component."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (17, 15), (63, 200), (64, 64), (65, 130), (200, 63), (129, 65), (200, 129)])
def test_plain_svst_at_tile_edges(m, n):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(1000 * m + n)
    k = min(m, n)
    r = (k + 1) // 2
    s = np.concatenate([np.linspace(9.0, 4.0, r), np.linspace(1.0, 0.5, k - r)])
    X = []
    for _ in range(2):
        q1, _ = np.linalg.qr(rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k)))
        q2, _ = np.linalg.qr(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))
        X.append(((q1 * s) @ q2.conj().T).astype(np.complex64))
    cm = torch.from_numpy(np.ascontiguousarray(np.stack(X).transpose(0, 2, 1))).cuda()
    out = np.transpose(M.svst_batch(cm, m, n, [2.0, 2.5], form=0).cpu().numpy(), (0, 2, 1))
    for x, o, beta in zip(X, out, (2.0, 2.5)):
        ref = O.svst(x.astype(np.complex128), beta)
        assert np.linalg.norm(o - ref) <= 2.4e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("ps,ss", [((16, 8, 8), (16, 8, 8)), ((4, 4, 4), (4, 4, 4)), ((6, 4, 3), (5, 4, 2))])
def test_gradient_at_tile_edges(ps, ss):
    """Gram sides 65 (tall: the split global patch, and overlapping patches of
    72 voxels) and 64 (wide patches of 65 frames)."""
    import torch
    import mslr_recon_b200 as M
    from mslr_recon_b200 import synth as S
    cfg = S.SynthConfig(N=(16, 8, 8), Nc=3, Nt=65, rank=3, frac=0.3, centre=2, seed=7,
                        patch_sizes=[list(ps)], strides=[list(ss)])
    pb = S.make_problem(cfg)
    prob = O.ReconProblem(smaps=pb["smaps"].astype(np.complex128), idx=pb["idx"],
                          y=pb["y"].astype(np.complex128), patch_sizes=pb["patch_sizes"], strides=pb["strides"])
    lam = [0.3 * v for v in prob.lambdas()]
    Xt = pb["x_true"].astype(np.complex128)
    loss_o, grad_o, X_o, restarts_o = O.pogm_unrolled_grad(prob, 5, Xt, lam, 1.0)
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(t).cuda()
    Nt, Nc, K = pb["y"].shape
    with M.MSLRContext(pb["N"], Nc, Nt, K, pb["patch_sizes"], pb["strides"], form="plain") as ctx:
        ctx.bind(dev(pb["smaps"], torch.complex64), dev(pb["y"], torch.complex64), dev(pb["idx"], torch.int32))
        ctx.set_lambdas(lam)
        loss, grad, X, restarts = ctx.pogm_grad(dev(pb["x_true"], torch.complex64), 5, 1.0)
    assert restarts == restarts_o
    assert O.rel_err(X.cpu().numpy(), X_o) < 1e-4
    assert loss == pytest.approx(loss_o, rel=1e-4)
    assert max(abs(g - o) for g, o in zip(grad, grad_o)) <= 1e-3 * max(abs(g) for g in grad_o)
