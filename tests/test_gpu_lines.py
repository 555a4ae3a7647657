"""The register-line SENSE kernels: every axis length with a compiled line
(5-smooth, 8 to 96) on each of the three axes, in the normal operator, the
encoding operator and its adjoint, against the FP64 oracle.

Tolerance: six transforms of up to about nine roundings a level over at most
seven levels, and the maps' two products, each 2^-24 relative; roundings add
up as their root, sqrt(6·9·7 + 10)·2^-24 = 1.2e-6 of the result."""
import numpy as np
import pytest

from oracle import mslr_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1.2e-6
TRIPLES = [(8, 9, 10), (12, 15, 16), (18, 20, 24), (25, 27, 30), (32, 36, 40), (45, 48, 50), (54, 60, 64),
           (72, 75, 80), (81, 90, 96)]
SHAPES = [t[k:] + t[:k] for t in TRIPLES for k in range(3)] + [(90, 90, 60), (48, 48, 32), (32, 32, 24)]


@pytest.mark.parametrize("N", SHAPES)
def test_every_line_length(N):
    import torch
    import mslr_recon_b200 as M
    Nx, Ny, Nz = N
    rng = np.random.default_rng(Nx * 10007 + Ny * 101 + Nz)
    nvox = Nx * Ny * Nz
    Nc, Nt = (9, 5) if nvox < 100000 else (3, 2)    # more than one coil group, an odd number of frames
    K = nvox // 5

    def cn(*shape):
        return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)

    smaps = cn(Nc, Nz, Ny, Nx)
    smaps /= np.sqrt(np.sum(np.abs(smaps) ** 2, axis=0))[None]
    idx = np.stack([np.sort(rng.choice(nvox, K, replace=False)) for _ in range(Nt)]).astype(np.int32)
    X, y = cn(2, Nt, Nz, Ny, Nx), cn(Nt, Nc, K)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rel = lambda a, b: np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b)
    s64 = smaps.astype(np.complex128)
    x64, y64 = X.astype(np.complex128), y.astype(np.complex128)
    fwd = O.sense_forward(x64.sum(axis=0), s64, idx)
    with M.MSLRContext(N, Nc, Nt, K, [list(N)], [list(N)]) as ctx:
        ctx.bind(dev(smaps), dev(y), dev(idx))
        assert rel(ctx.forward(dev(X[0])), O.sense_forward(x64[0], s64, idx)) < TOL
        assert rel(ctx.adjoint(dev(y)), O.sense_adjoint(y64, s64, idx)) < TOL
        assert rel(ctx.normal(dev(X)), O.sense_adjoint(fwd - y64, s64, idx)) < TOL
        assert rel(ctx.normal(dev(X[0]), subtract_data=False),
                   O.sense_adjoint(O.sense_forward(x64[0], s64, idx), s64, idx)) < TOL
