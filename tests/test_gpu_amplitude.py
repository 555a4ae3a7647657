"""The eigen stage at any amplitude of its input: SVST(aX, aβ) = a SVST(X, β) and
‖aX‖_* = a ‖X‖_*.

For a power of two a nothing on the way rounds differently (Gram, T, its
eigenvalues, W and the rebuild scale by powers of two), so those results are
equal bit for bit; at 1e-8 … 1e6 they are compared with matrices whose SVST is
known in closed form, X = Q₁ diag(s) Q₂ᴴ, SVST = Q₁ diag(max(s − β, 0)) Q₂ᴴ.
Tolerance there: split-BF16 Gram, W and rebuild, 3·2^-17 of a product left out
each and as much for the soft threshold's factor: 4·3·2^-17 = 9.2e-5.  Sides
of every kernel of the tridiagonalisation."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu

SIDES = [5, 8, 20, 64, 90, 100, 128, 130, 300, 301, 400]
POWERS = [-30, -20, -13, 14, 20, 40]


def cn(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


def stack_of(rng, n):
    """A static series with noise, low rank, full rank, columns that differ by
    1e-5 in size, one nonzero column, zeros."""
    m = n + 40
    static = np.outer(cn(rng, m), np.exp(0.05j * rng.standard_normal(n)))
    graded = cn(rng, m, n)
    graded[:, n // 2:] *= 1e-5
    one = np.zeros((m, n), complex)
    one[:, 3] = cn(rng, m)
    stack = [static + 1e-3 * cn(rng, m, n), cn(rng, m, 4) @ cn(rng, 4, n), cn(rng, m, n), graded, one,
             np.zeros((m, n), complex)]
    return np.stack(stack).astype(np.complex64), [0.5, 3.0, 0.7 * np.sqrt(m), 2.0, 1.0, 1.0]


@pytest.mark.parametrize("n", SIDES)
def test_powers_of_two_scale_the_result(n):
    import torch
    import mslr_recon_b200 as M
    X, betas = stack_of(np.random.default_rng(n), n)
    m = X.shape[1]
    cm = torch.from_numpy(np.ascontiguousarray(X.transpose(0, 2, 1))).cuda()
    unit = M.svst_batch(cm, m, n, betas)
    assert bool(torch.isfinite(torch.view_as_real(unit)).all())
    for e in POWERS:
        a = 2.0 ** e
        out = M.svst_batch(cm * a, m, n, [a * b for b in betas])
        assert torch.equal(out, unit * a), e


@pytest.mark.parametrize("a", [1e-8, 1e-4, 1.0, 1e4, 1e6])
@pytest.mark.parametrize("n", SIDES)
def test_closed_form_at_amplitude(n, a):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(7 * n)
    m = n + 40
    q1, _ = np.linalg.qr(cn(rng, m, n))
    q2, _ = np.linalg.qr(cn(rng, n, n))
    out, ref = [], []
    for r in (3, n // 2):
        s = np.concatenate([np.linspace(9.0, 4.0, r), np.linspace(1.0, 0.5, n - r)])
        X = a * (q1 * s) @ q2.conj().T
        ref.append(a * (q1 * np.maximum(s - 2.0, 0.0)) @ q2.conj().T)
        out.append(M.SVST(torch.from_numpy(X.astype(np.complex64)).cuda(), 2.0 * a).cpu().numpy())
    for o, w in zip(out, ref):
        assert np.linalg.norm(o - w) <= 9.2e-5 * np.linalg.norm(w)


@pytest.mark.parametrize("n", SIDES)
def test_columns_of_very_different_size(n):
    """A trailing block whose Gram is 1e-22 of the leading one's."""
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(11 * n)
    X = cn(rng, n + 40, n)
    X[:, n // 2:] *= 1e-11
    X = X.astype(np.complex64)
    out = M.SVST(torch.from_numpy(X).cuda(), 2.0).cpu().numpy()
    ref = O.svst(X.astype(np.complex128), 2.0)
    assert np.linalg.norm(out - ref) <= 9.2e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("tiny", [1e-12, 1e-17, 1e-20, 1e-35])
@pytest.mark.parametrize("n", SIDES)
def test_rows_that_have_faded(n, tiny):
    """Rows down to 1e-35, as thresholded voxels outside the object have: the
    squares of what couples them leave FP32."""
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(13 * n)
    X = cn(rng, n, n + 70)
    X[n - 2] *= 1e-13
    X[n - 1] *= tiny
    X[:, ::7] *= tiny
    X = X.astype(np.complex64)
    out = M.SVST(torch.from_numpy(X).cuda(), 2.0).cpu().numpy()
    ref = O.svst(X.astype(np.complex128), 2.0)
    assert np.linalg.norm(out - ref) <= 9.2e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("Nt", [20, 64, 128, 300])
def test_nuclear_norm_scales(Nt):
    """The values-only mode, on a global patch and on local ones."""
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(Nt)
    N = (12, 10, 8)
    img = np.exp(1j * rng.standard_normal((1, 8, 10, 12))) + 0.05 * cn(rng, Nt, 8, 10, 12)
    x = torch.from_numpy(img.astype(np.complex64)).cuda()
    with M.MSLRContext(N, 1, Nt, 1, [[12, 10, 8], [6, 5, 4]], [[12, 10, 8], [6, 5, 4]]) as ctx:
        for s in (0, 1):
            unit = ctx.patch_nucnorm(s, x)
            assert unit > 0.0
            for e in POWERS:
                assert ctx.patch_nucnorm(s, x * 2.0 ** e) == unit * 2.0 ** e, (s, e)


def test_gradient_with_an_almost_empty_background():
    """All eigenpairs of patches whose values are 1e-12 of the others'.  The
    gradient carries FP32 rounding of about 1e-5 over a few iterations."""
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(3)
    N, Nc, Nt = (16, 16, 8), 2, 40
    nvox = 16 * 16 * 8
    smaps = cn(rng, Nc, 8, 16, 16)
    smaps /= np.sqrt((np.abs(smaps) ** 2).sum(0))
    y = cn(rng, Nt, Nc, nvox).astype(np.complex64)
    idx = np.tile(np.arange(nvox, dtype=np.int32), (Nt, 1))
    Xt = cn(rng, Nt, 8, 16, 16).astype(np.complex64)
    Xt[..., 8:] = 0

    def grad(background):
        s = smaps.copy()
        s[..., 8:] *= background
        with M.MSLRContext(N, Nc, Nt, nvox, [[8, 8, 8]], [[8, 8, 8]]) as ctx:
            ctx.bind(*(torch.from_numpy(v).cuda() for v in (s.astype(np.complex64), y, idx)))
            ctx.set_lambdas([10.0])
            loss, g, _, _ = ctx.pogm_grad(torch.from_numpy(Xt).cuda(), 3, 1.0)
            return loss, g[0]

    loss, g = grad(1e-12)
    loss0, g0 = grad(0.0)   # what the background contributes is far below that rounding
    assert g0 != 0.0 and abs(loss - loss0) <= 1e-6 * loss0 and abs(g - g0) <= 1e-4 * abs(g0)
