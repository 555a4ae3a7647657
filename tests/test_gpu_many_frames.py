"""More frames than one dimension of a grid holds (65 535): the binding and the
SENSE operators at the first, last and some other frames, against the FP64
oracle; tolerance as for other line lengths, 1.2e-6."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu


def test_70000_frames():
    import torch
    import mslr_recon_b200 as M
    N, Nc, Nt, K = (8, 8, 8), 4, 70000, 16
    cn = lambda *s: torch.view_as_complex(torch.randn(s + (2,), generator=gen, device="cuda"))
    gen = torch.Generator(device="cuda").manual_seed(5)
    smaps, y, x = cn(Nc, 8, 8, 8), cn(Nt, Nc, K), cn(Nt, 8, 8, 8)
    idx = torch.sort(torch.rand((Nt, 512), generator=gen, device="cuda").argsort(1)[:, :K]).values.int().contiguous()
    some = [0, 1, 35000, 65535, 65536, Nt - 1]
    s64 = smaps.cpu().numpy().astype(np.complex128)
    at = lambda t: t[some].cpu().numpy()
    with M.MSLRContext(N, Nc, Nt, K, [[4, 4, 4]], [[4, 4, 4]]) as ctx:
        ctx.bind(smaps, y, idx)
        got = {"fwd": ctx.forward(x), "adj": ctx.adjoint(y), "normal": ctx.normal(x)}
        x64, y64, i = at(x).astype(np.complex128), at(y).astype(np.complex128), at(idx)
        fwd = O.sense_forward(x64, s64, i)
        want = {"fwd": fwd, "adj": O.sense_adjoint(y64, s64, i), "normal": O.sense_adjoint(fwd - y64, s64, i)}
        for k in want:
            assert np.linalg.norm(at(got[k]) - want[k]) <= 1.2e-6 * np.linalg.norm(want[k]), k
