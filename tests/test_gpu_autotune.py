"""The autotuner times the shape that the context starts with as well: what it
keeps is not slower.  Five coils, which it used to split into groups of three
and two (9 % slower here); 4 % for the clock's noise, the least of seven runs a
side."""
import pytest

pytestmark = pytest.mark.gpu


def test_not_slower_than_the_default():
    import torch
    import mslr_recon_b200 as M
    N, Nc, Nt = (75, 64, 45), 5, 24
    nvox = 75 * 64 * 45
    K = nvox // 6
    gen = torch.Generator(device="cuda").manual_seed(0)
    cn = lambda *s: torch.view_as_complex(torch.randn(s + (2,), generator=gen, device="cuda"))
    idx = torch.stack([torch.randperm(nvox, generator=gen, device="cuda")[:K].sort().values for _ in range(Nt)]).int()

    def least(ctx, X):
        best = float("inf")
        for _ in range(7):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            ctx.normal(X)
            a.record()
            for _ in range(10):
                ctx.normal(X)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    with M.MSLRContext(N, Nc, Nt, K, [list(N)], [list(N)]) as ctx:
        ctx.bind(cn(Nc, 45, 64, 75), cn(Nt, Nc, K), idx)
        X = cn(Nt, 45, 64, 75)
        before = least(ctx, X)
        ctx.autotune()
        assert least(ctx, X) <= 1.04 * before
