"""Device memory of the register-line SENSE form: the buffer of the summed image,
one more image series, is there only once a call needs it (from the binding on
in a context of several scales), also when that call is being captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, NC, NT, K = (12, 15, 10), 10, 6, 400
NVOX = 12 * 15 * 10
SERIES = NT * NVOX * 8


def inputs():
    import torch
    rng = np.random.default_rng(0)
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()
    idx = np.stack([np.sort(rng.choice(NVOX, K, replace=False)) for _ in range(NT)]).astype(np.int32)
    return (cn(NC, 10, 15, 12), cn(NT, NC, K), torch.from_numpy(idx).cuda()), cn(2, NT, 10, 15, 12)


def grown(ctx, call):
    before = ctx.workspace_bytes()
    call()
    return ctx.workspace_bytes() - before


def plain_binding(data, sizes):
    """What binding takes in the plain form, which has no such buffer."""
    import mslr_recon_b200 as M
    with M.MSLRContext(N, NC, NT, K, sizes, sizes, form="plain") as ctx:
        return grown(ctx, lambda: ctx.bind(*data))


def test_one_scale():
    import mslr_recon_b200 as M
    data, X = inputs()
    bound = plain_binding(data, [list(N)])
    with M.MSLRContext(N, NC, NT, K, [list(N)], [list(N)]) as ctx:
        assert grown(ctx, lambda: ctx.bind(*data)) == bound
        assert grown(ctx, lambda: ctx.normal(X[0])) == 0
        assert grown(ctx, lambda: ctx.normal(X)) == SERIES
        assert grown(ctx, lambda: ctx.normal(X)) == 0


def test_two_scales():
    import mslr_recon_b200 as M
    data, X = inputs()
    bound = plain_binding(data, [list(N), [6, 5, 5]])
    with M.MSLRContext(N, NC, NT, K, [list(N), [6, 5, 5]], [list(N), [6, 5, 5]]) as ctx:
        assert grown(ctx, lambda: ctx.bind(*data)) == bound + SERIES
        assert grown(ctx, lambda: ctx.normal(X)) == 0


def test_first_use_under_capture():
    import torch
    import mslr_recon_b200 as M
    data, X = inputs()
    with M.MSLRContext(N, NC, NT, K, [list(N)], [list(N)]) as ctx:
        ctx.bind(*data)
        out = torch.empty_like(X[0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ctx.normal(X, out=out)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ctx.normal(X))
        del graph
