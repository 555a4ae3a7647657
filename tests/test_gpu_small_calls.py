"""Small SENSE calls: up to 16 MB of k-space (64 with more than eight coils), each
pass is one launch, whatever the coils and frames; on both sides of that border
the operators agree with the FP64 oracle, to 1.2e-6 as for every line length."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu


def bound(N, Nc, Nt, rng):
    import torch
    import mslr_recon_b200 as M
    nvox = N[0] * N[1] * N[2]
    K = nvox // 4
    cn = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    smaps, y = cn(Nc, *N[::-1]), cn(Nt, Nc, K)
    smaps /= np.sqrt((np.abs(smaps) ** 2).sum(0))
    idx = np.sort(rng.random((Nt, nvox)).argsort(1)[:, :K], 1).astype(np.int32)
    ctx = M.MSLRContext(N, Nc, Nt, K, [[8, 8, 8]], [[8, 8, 8]])
    ctx.bind(*(torch.from_numpy(v).cuda() for v in (smaps, y, idx)))
    return ctx, smaps, y, idx, cn(Nt, *N[::-1])


@pytest.mark.parametrize("N,Nc,Nt,passes", [((12, 12, 12), 16, 1, 6), ((12, 12, 12), 32, 3, 6), ((12, 12, 12), 1, 40, 6),
                                            ((16, 16, 16), 4, 15, 6), ((32, 32, 24), 16, 20, 4), ((48, 48, 32), 4, 6, 4)])
def test_one_launch_a_pass(N, Nc, Nt, passes):
    import torch
    ctx, _, y, _, x = bound(N, Nc, Nt, np.random.default_rng(1))
    with ctx:
        xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        for call, most in ((lambda: ctx.normal(xd), passes), (lambda: ctx.forward(xd), passes),
                           (lambda: ctx.adjoint(yd), passes)):
            before = ctx.launch_count()
            call()
            assert ctx.launch_count() - before <= most


@pytest.mark.parametrize("N,Nc", [((8, 8, 8), 1), ((8, 8, 8), 16), ((16, 16, 16), 8), ((80, 8, 8), 4), ((48, 45, 40), 2)])
def test_one_frame_of_a_small_image(N, Nc):
    """Three launches, not one a pass of the lines."""
    import torch
    ctx, _, y, _, x = bound(N, Nc, 1, np.random.default_rng(2))
    with ctx:
        xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        for call in (lambda: ctx.normal(xd), lambda: ctx.forward(xd), lambda: ctx.adjoint(yd)):
            before = ctx.launch_count()
            call()
            assert ctx.launch_count() - before <= 3


@pytest.mark.parametrize("N,Nc,Nt", [((20, 18, 16), 8, 43), ((20, 18, 16), 8, 44), ((20, 18, 16), 12, 115),
                                     ((20, 18, 16), 12, 116), ((8, 8, 8), 1, 1), ((8, 8, 8), 1, 2), ((8, 8, 8), 20, 1), ((8, 8, 8), 24, 1), ((24, 20, 18), 8, 1),
                                     ((24, 20, 18), 9, 1), ((20, 24, 50), 4, 1), ((20, 24, 54), 4, 1), ((64, 64, 40), 2, 1),
                                     ((64, 72, 16), 2, 1)])
def test_both_sides_of_each_border(N, Nc, Nt):
    """15.9 and 16.2 MB, 63.6 and 64.1; one and two frames; one frame of 8 and 9
    coils, on planes of 4096 points and more, and of fewer and more points."""
    import torch
    ctx, smaps, y, idx, x = bound(N, Nc, Nt, np.random.default_rng(Nt))
    s64, x64, y64 = smaps.astype(np.complex128), x.astype(np.complex128), y.astype(np.complex128)
    fwd = O.sense_forward(x64, s64, idx)
    with ctx:
        xd = torch.from_numpy(x).cuda()
        for got, want in ((ctx.forward(xd), fwd), (ctx.adjoint(torch.from_numpy(y).cuda()), O.sense_adjoint(y64, s64, idx)),
                          (ctx.normal(xd), O.sense_adjoint(fwd - y64, s64, idx))):
            assert np.linalg.norm(got.cpu().numpy() - want) <= 1.2e-6 * np.linalg.norm(want)
