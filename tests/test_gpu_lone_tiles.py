"""Grams of no more tiles than SMs, in chunks of 32 elements: contractions around
one and two chunks and long ones, sides around 64 and the 128-wide tile, 148
tiles and 149, wide patches, against matrices whose SVST is known in closed
form, X = Q₁ diag(s) Q₂ᴴ, SVST = Q₁ diag(max(s − β, 0)) Q₂ᴴ.

Tolerance: the products leave out 3·2^-17 (split BF16) or 2·2^-12 (TF32) of
Gram, W and rebuild each, and as much again for the soft threshold's factor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {1: 4 * 3 * 2.0 ** -17, 2: 4 * 2 * 2.0 ** -12}


def cn(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


@pytest.mark.parametrize("form", [1, 2])
@pytest.mark.parametrize("m,n,batch", [(31, 16, 1), (32, 16, 3), (33, 16, 1), (63, 20, 1), (64, 20, 1), (65, 20, 1), (20, 65, 1),
                                       (95, 64, 148), (97, 64, 149), (161, 65, 1), (500, 128, 2), (515, 129, 49),
                                       (515, 129, 50), (129, 1031, 1), (20001, 40, 1)])
def test_values(m, n, batch, form):
    import torch
    import mslr_recon_b200 as M
    rng = np.random.default_rng(m * n)
    k = min(m, n)
    q1, q2 = np.linalg.qr(cn(rng, m, k))[0], np.linalg.qr(cn(rng, n, k))[0]
    r = k // 2
    s = np.concatenate([np.linspace(9.0, 4.0, r), np.linspace(1.0, 0.5, k - r)])
    scale = rng.uniform(0.5, 2.0, batch)
    X = ((q1 * s) @ q2.conj().T).astype(np.complex64)
    ref = (q1 * np.maximum(s - 2.0, 0.0)) @ q2.conj().T
    cm = torch.from_numpy(np.stack([np.ascontiguousarray((np.float32(c) * X).T) for c in scale])).cuda()
    out = M.svst_batch(cm, m, n, [2.0 * float(np.float32(c)) for c in scale], form=form).cpu().numpy()
    for b, c in enumerate(scale):
        assert np.linalg.norm(out[b].T - c * ref) <= TOL[form] * np.linalg.norm(c * ref), b


def test_one_tall_matrix():
    """100 000 x 128, whose Gram is one tile on one SM and nearly the whole call:
    5.7 ms at 1965 MHz, 7.6 in chunks of 16.  Normalised by the measured FP32
    rate for the clock (70 TFLOP/s there); between the two."""
    import torch
    import mslr_recon_b200 as M
    from mslr_recon_b200.context import fp32_peak
    X = torch.view_as_complex(torch.randn((1, 128, 100000, 2), device="cuda"))
    best = float("inf")
    for _ in range(5):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        M.svst_batch(X, 100000, 128, [100.0])
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    assert best * fp32_peak() / 70.0 <= 6.7
