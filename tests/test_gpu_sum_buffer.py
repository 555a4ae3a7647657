"""Device memory of the register-line SENSE form: the image that several scales
sum to has no buffer of its own.  A context of one scale is less than an image
series larger than in the plain form (its sample bits), and binding and the
normal operator take what they take there; the sum may be part of a captured
call, and does not disturb an iteration that it comes between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, NC, NT, K = (12, 15, 10), 10, 6, 400
SCALES = {1: [list(N)], 2: [list(N), [6, 5, 5]]}


def inputs():
    import torch
    rng = np.random.default_rng(0)
    cn = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()
    nvox = 12 * 15 * 10
    idx = np.stack([np.sort(rng.choice(nvox, K, replace=False)) for _ in range(NT)]).astype(np.int32)
    return (cn(NC, 10, 15, 12), cn(NT, NC, K), torch.from_numpy(idx).cuda()), cn(2, NT, 10, 15, 12)


def context(scales, form="tuned"):
    import mslr_recon_b200 as M
    return M.MSLRContext(N, NC, NT, K, SCALES[scales], SCALES[scales], form=form)


@pytest.mark.parametrize("scales", [1, 2])
def test_memory(scales):
    data, X = inputs()
    made, grown = {}, {}
    for form in ("plain", "tuned"):
        with context(scales, form) as ctx:
            before = made[form] = ctx.workspace_bytes()
            ctx.bind(*data)
            ctx.normal(X)
            Y = X[0].clone()
            ctx.normal(Y, out=Y)
            grown[form] = ctx.workspace_bytes() - before
    assert grown["tuned"] == grown["plain"]
    if scales == 1:   # (with more, the tuned form has an SVST workspace for each)
        assert made["tuned"] - made["plain"] < NT * 12 * 15 * 10 * 8


def test_under_capture():
    import torch
    data, X = inputs()
    with context(1) as ctx:
        ctx.bind(*data)
        out = torch.empty_like(X[0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ctx.normal(X, out=out)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ctx.normal(X))
        del graph


@pytest.mark.parametrize("bsig", [1.0, 0.7])
def test_between_the_steps_of_an_iteration(bsig):
    import torch
    data, X = inputs()
    runs = []
    for between in (False, True):
        with context(2) as ctx:
            ctx.bind(*data)
            x = ctx.init_x0()
            ctx.pogm_begin(x, 4, 2.0, bsig=bsig)
            for _ in range(4):
                ctx.pogm_step(x)
                if between:
                    ctx.normal(X)
                    Y = X[0].clone()
                    ctx.normal(Y, out=Y)
                    ctx.cost(X)
            runs.append((x, ctx.pogm_restarts()))
    assert torch.equal(runs[0][0], runs[1][0]) and runs[0][1] == runs[1][1]
