"""The work that users of this framework have it do, as cases to be timed.

A reconstruction is: coil maps, sampled k-space and sample positions are bound
to a context, POGM iterates (SENSE normal operator, patch SVST per scale, the
update), and the images come back.  The cases are those calls and the blocks
they consist of, each through a public entry point, from one small SVST to
iterations at the full fMRI volume.  All inputs are made on the GPU from the
seed: low-rank image series with noise, smooth coil maps, random sampling with
a fully sampled centre, scaled as run_recon scales its data.
"""
from __future__ import annotations

import math

import torch

import mslr_recon_b200 as M
from mslr_recon_b200 import recon as R

DEV = "cuda"
C64, C128 = torch.complex64, torch.complex128


# --------------------------------------------------------------------------
# The cases.  nx, ny, nz: image; nc: coils; nt: frames; p, s: side and stride
# of the local patches (0: none; the global patch is one of the scales of the
# whole calls); keep: "all" thresholds below every singular value (the
# λ_k of a well-scaled series: full rank), "signal" thresholds at the noise's
# largest singular value, so that the low-rank part stays.
# --------------------------------------------------------------------------
def listed():
    return [
        # one matrix on its own: the smallest call, latency and launches
        dict(name="svst_one_216x64", kind="svst", m=216, n=64, batch=1, keep="signal"),
        # a stack of ordinary patches handed over as matrices, thresholded
        # below the spectrum
        dict(name="svst_stack_512x128", kind="svst", m=512, n=128, batch=40, keep="all"),
        # patchSVST on an image with no context, half-overlapping patches that
        # do not fit the odd image: extract, threshold, recombine
        dict(name="patchsvst_ragged", kind="patchsvst", nx=35, ny=29, nz=21, nt=50, p=7, s=4, keep="signal"),
        # one scale of the prox at the fMRI volume: 486 patches of 1000 x 300,
        # every singular value above the threshold
        dict(name="prox_fmri_10", kind="prox", nx=90, ny=90, nz=60, nt=300, p=10, s=10, keep="all"),
        # the same with half-overlapping small patches, many more of them than
        # of the others, thresholded at the noise
        dict(name="prox_overlap_6", kind="prox", nx=48, ny=48, nz=32, nt=128, p=6, s=3, keep="signal"),
        # the SENSE normal operator (gradient of the data term): a small study
        dict(name="normal_small", kind="normal", nx=32, ny=32, nz=24, nc=8, nt=64, ns=1),
        # at a volume whose axes have odd factors, two scales summed
        dict(name="normal_odd", kind="normal", nx=75, ny=64, nz=45, nc=12, nt=40, ns=2),
        # at the fMRI volume with its 18 coils and 300 frames
        dict(name="normal_fmri", kind="normal", nx=90, ny=90, nz=60, nc=18, nt=300, ns=2),
        # the encoding operator and its adjoint (simulation, residuals)
        dict(name="encode_decode_fmri", kind="sense", nx=90, ny=90, nz=60, nc=18, nt=24),
        # a small reconstruction of 20 iterations, one local scale
        dict(name="recon_small", kind="recon", nx=32, ny=32, nz=24, nc=8, nt=64, ng=0, p=6, s=6, niter=20),
        # iterations at the fMRI volume: global and 10^3 scales
        dict(name="recon_fmri", kind="recon", nx=90, ny=90, nz=60, nc=18, nt=300, ng=1, p=10, s=10, niter=3),
        # the backward direction: gradient of a short unrolled reconstruction
        # with respect to the scales' weights
        dict(name="grad_unrolled", kind="grad", nx=48, ny=48, nz=32, nc=12, nt=128, ng=1, p=8, s=8, niter=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


AXES = (24, 30, 32, 36, 40, 45, 48, 54, 60, 64, 72, 75, 80, 90)   # image sides that scanners are set to


def draw(rng):
    kind = rng.choice(["svst", "patchsvst", "prox", "normal", "normal", "sense", "recon", "grad"])
    keep = rng.choice(["all", "signal"])
    if kind == "svst":
        m, n = _log_int(rng, 27, 1000), _log_int(rng, 12, 300)
        if rng.random() < 0.25:
            m, n = n, m
        return dict(kind=kind, m=m, n=n, batch=_log_int(rng, 1, 64), keep=keep)
    if kind == "patchsvst":
        return dict(kind=kind, nx=rng.randint(16, 40), ny=rng.randint(16, 40), nz=rng.randint(12, 32),
                    nt=_log_int(rng, 16, 128), p=rng.randint(4, 8), s=rng.randint(3, 8), keep=keep)
    if kind == "prox":
        p = rng.randint(5, 10)
        return dict(kind=kind, nx=rng.choice(AXES[1:9]), ny=rng.choice(AXES[1:9]), nz=rng.choice(AXES[:6]),
                    nt=_log_int(rng, 32, 300), p=p, s=rng.choice([p, (p + 1) // 2]), keep=keep)
    shape = rng.choice([(90, 90, 60), (48, 48, 32), (32, 32, 24), None, None])
    if shape is None:
        shape = (rng.choice(AXES), rng.choice(AXES), rng.choice(AXES[:9]))
    nx, ny, nz = shape
    nc, nt = rng.randint(4, 20), _log_int(rng, 8, 100)
    if kind == "normal":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nc=nc, nt=nt, ns=rng.randint(1, 3))
    if kind == "sense":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nc=nc, nt=min(nt, 24))
    p = rng.randint(5, 10)
    if kind == "recon":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nc=nc, nt=nt, ng=rng.randint(0, 1), p=p, s=p,
                    niter=rng.randint(2, 8))
    return dict(kind=kind, nx=rng.choice(AXES[:5]), ny=rng.choice(AXES[:5]), nz=rng.choice((12, 15, 16, 20, 24)),
                nc=rng.randint(3, 8), nt=rng.randint(12, 64), ng=rng.randint(0, 1), p=rng.randint(4, 6), s=4,
                niter=rng.randint(2, 4))


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
NOISE = 0.05   # image noise relative to the series' rms


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(0x5EED0000 + int(seed))
    return g


def _cn(g, *shape, dtype=C64):
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def _series(g, nt, nvox, rank=8):
    """Low-rank image series (nt, nvox) of unit rms with noise."""
    rank = min(rank, nt)
    basis, _ = torch.linalg.qr(_cn(g, nt, rank, dtype=C128))
    maps = _cn(g, rank, nvox)
    x = basis.to(C64) @ maps
    x *= math.sqrt(nt / rank)
    for t in range(0, nt, 64):
        x[t:t + 64] += NOISE * _cn(g, min(64, nt - t), nvox)
    return x


def _stack(c, seed):
    """(batch, n, m) memory of `batch` column-major m x n matrices."""
    g = _gen(seed)
    return torch.stack([_series(g, c["n"], c["m"], 4) for _ in range(c["batch"])]).contiguous()


def _threshold(keep, m, n, noise=NOISE):
    if keep == "signal":   # the noise's largest singular value, with a margin
        return 1.05 * noise * (math.sqrt(m) + math.sqrt(n))
    return 0.2 * noise * abs(math.sqrt(m) - math.sqrt(n)) + 1e-3


def _coil_maps(g, nx, ny, nz, nc):
    z, y, x = torch.meshgrid(*(torch.linspace(-1, 1, n, device=DEV, dtype=torch.float64) for n in (nz, ny, nx)),
                             indexing="ij")
    maps = torch.empty((nc, nz, ny, nx), dtype=C64, device=DEV)
    par = torch.randn((nc, 4), generator=g, device=DEV, dtype=torch.float64).cpu()
    for c in range(nc):   # smooth bumps on a sphere around the volume, each with a linear phase
        zc = 1 - 2 * (c + 0.5) / nc
        rc, th = math.sqrt(max(0.0, 1 - zc * zc)), math.pi * (3 - math.sqrt(5)) * c
        d2 = (x - 1.3 * rc * math.cos(th)) ** 2 + (y - 1.3 * rc * math.sin(th)) ** 2 + (z - 1.3 * zc) ** 2
        ph = 0.5 * (float(par[c, 0]) * x + float(par[c, 1]) * y + float(par[c, 2]) * z) + math.pi * float(par[c, 3])
        maps[c] = torch.polar(torch.exp(-d2 / 1.28), ph).to(C64)
    maps /= maps.abs().square().sum(0).sqrt()
    return maps


def _samples(g, nx, ny, nz, nt, frac=1 / 6):
    """Ascending sample positions (nt, K): a fully sampled centre and random points."""
    nvox = nx * ny * nz
    side = [min(12, n // 4) for n in (nx, ny, nz)]
    lo = [n // 2 - k // 2 for n, k in zip((nx, ny, nz), side)]
    centre = torch.zeros((nz, ny, nx), dtype=torch.bool, device=DEV)
    centre[lo[2]:lo[2] + side[2], lo[1]:lo[1] + side[1], lo[0]:lo[0] + side[0]] = True
    centre = centre.reshape(-1)
    K = max(int(round(frac * nvox)), int(centre.sum()))
    idx = torch.empty((nt, K), dtype=torch.int32, device=DEV)
    for t in range(nt):
        key = torch.rand(nvox, generator=g, device=DEV)
        key[centre] = -1.0
        idx[t] = torch.topk(key, K, largest=False, sorted=False).indices.sort().values.to(torch.int32)
    return idx


AX = (-3, -2, -1)


def _fwd(x, maps, idx):
    """Centred unitary encoding of one frame: (nc, K)."""
    k = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(maps * x, dim=AX), dim=AX, norm="ortho"), dim=AX)
    return k.reshape(maps.shape[0], -1)[:, idx.long()]


def _adj(y, maps, idx):
    k = torch.zeros((maps.shape[0], maps[0].numel()), dtype=y.dtype, device=DEV)
    k[:, idx.long()] = y
    im = torch.fft.ifftn(torch.fft.ifftshift(k.reshape(maps.shape), dim=AX), dim=AX, norm="ortho")
    return (maps.conj() * torch.fft.fftshift(im, dim=AX)).sum(0)


def _acquisition(c, seed):
    """(maps, idx, y, x): a scaled acquisition of a low-rank series."""
    g = _gen(seed)
    nx, ny, nz, nt = c["nx"], c["ny"], c["nz"], c["nt"]
    maps = _coil_maps(g, nx, ny, nz, c["nc"])
    idx = _samples(g, nx, ny, nz, nt)
    x = _series(g, nt, nx * ny * nz).reshape(nt, nz, ny, nx)
    y = torch.empty((nt, c["nc"], idx.shape[1]), dtype=C64, device=DEV)
    mags = []
    for t in range(nt):
        y[t] = _fwd(x[t], maps, idx[t])
        y[t] += 0.01 * _cn(g, *y.shape[1:])
        if t < 4:   # run_recon divides by the 99th percentile of the combined image
            mags.append(_adj(y[t], maps, idx[t]).abs().reshape(-1) / math.sqrt(nx * ny * nz))
    mag = torch.cat(mags)
    scale = float(mag.kthvalue(int(0.99 * mag.numel())).values)
    y /= scale
    x /= scale
    return maps, idx, y, x


def _scales(c):
    vol = [c["nx"], c["ny"], c["nz"]]
    ps = [vol] * c.get("ng", 1) + ([[c["p"]] * 3] if c.get("p") else [])
    ss = [vol] * c.get("ng", 1) + ([[c["s"]] * 3] if c.get("p") else [])
    return ps, ss


def _dims(c):
    return (c["nx"], c["ny"], c["nz"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "svst":
        X = _stack(c, seed)
        if c["batch"] == 1:
            return dict(c=c, X=X[0].t().contiguous(), beta=_threshold(c["keep"], c["m"], c["n"]))
        return dict(c=c, X=X, betas=[_threshold(c["keep"], c["m"], c["n"])] * c["batch"])
    if kind in ("patchsvst", "prox"):
        img = _series(_gen(seed), c["nt"], math.prod(_dims(c))).reshape(c["nt"], c["nz"], c["ny"], c["nx"])
        beta = _threshold(c["keep"], c["p"] ** 3, c["nt"])
        if kind == "patchsvst":
            return dict(c=c, img=img, beta=beta)
        ctx = M.MSLRContext(_dims(c), 1, c["nt"], 1, [[c["p"]] * 3], [[c["s"]] * 3])
        return dict(c=c, img=img, beta=beta, ctx=ctx)
    maps, idx, y, x = _acquisition(c, seed)
    ps, ss = _scales(c) if kind in ("recon", "grad") else ([list(_dims(c))], [list(_dims(c))])
    ctx = M.MSLRContext(_dims(c), c["nc"], c["nt"], idx.shape[1], ps, ss)
    ctx.bind(maps, y, idx)
    if kind == "normal":
        X = torch.stack([x / c["ns"]] * c["ns"])
        X[0].mul_(0.9)
        return dict(c=c, ctx=ctx, X=X)
    if kind == "sense":
        return dict(c=c, ctx=ctx, x=x, y=y)
    # σ₁(A) <= 1 for normalised maps, as users who skip the power iteration set it
    st = dict(c=c, ctx=ctx, L=float(ctx.Ns), X=torch.empty(ctx.x_shape, dtype=C64, device=DEV))
    if kind == "grad":
        st["x_true"] = x
    return st


def run(st):
    c = st["c"]
    kind = c["kind"]
    if kind == "svst":
        if c["batch"] == 1:
            return R.SVST(st["X"], st["beta"])
        return R.svst_batch(st["X"], c["m"], c["n"], st["betas"])
    if kind == "patchsvst":
        return R.patchSVST(st["img"], st["beta"], [c["p"]] * 3, [c["s"]] * 3)
    if kind == "prox":
        return st["ctx"].patch_svst(0, st["beta"], st["img"])
    if kind == "normal":
        return st["ctx"].normal(st["X"])
    if kind == "sense":
        return {"y": st["ctx"].forward(st["x"]), "x": st["ctx"].adjoint(st["y"])}
    if kind == "recon":
        X = st["ctx"].init_x0(st["X"])
        return {"X": X, "restarts": st["ctx"].pogm_run(X, c["niter"], st["L"])}
    loss, grad, X, restarts = st["ctx"].pogm_grad(st["x_true"], c["niter"], st["L"], X=st["X"])
    return {"loss": loss, "grad": grad, "X": X, "restarts": restarts}


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _starts(n, p, s):
    p = min(p, n)
    return [min(i * s, n - p) for i in range(-(-(n - p) // s) + 1)]


def _svst_flops(m, n):
    """Gram, eigenpairs of a k x k Hermitian matrix, rebuild (complex: 8 flops a multiply-add)."""
    k, big = min(m, n), max(m, n)
    return 4.0 * k * k * big + 8.0 * 4 / 3 * k ** 3 + 8.0 * k ** 3 + 8.0 * k * k * big


def _prox_flops(dims, nt, p, s):
    ps = [min(a, b) for a, b in zip(p, dims)]
    npatch = math.prod(len(_starts(n, a, b)) for n, a, b in zip(dims, p, s))
    return npatch * _svst_flops(math.prod(ps), nt)


def work(case):
    c, kind = case, case["kind"]
    if kind == "svst":
        return dict(bytes=16.0 * c["m"] * c["n"] * c["batch"], flops=c["batch"] * _svst_flops(c["m"], c["n"]))
    nvox, nt = math.prod(_dims(c)), c["nt"]
    image = 8.0 * nvox * nt
    if kind in ("patchsvst", "prox"):
        return dict(bytes=2 * image, flops=_prox_flops(_dims(c), nt, [c["p"]] * 3, [c["s"]] * 3))
    nc, K = c["nc"], round(nvox / 6)
    maps = 8.0 * nc * nvox
    fft = 5.0 * nvox * math.log2(nvox) * nc * nt
    pt = 8.0 * 2 * nvox * nc * nt   # the multiplications by the maps and their conjugates
    if kind == "normal":
        # images in, A'y and the gradient, maps, mask
        return dict(bytes=(c["ns"] + 2) * image + maps + nvox * nt / 8, flops=2 * fft + pt)
    if kind == "sense":
        return dict(bytes=2 * image + 2 * (8.0 * nc * K * nt) + 2 * 4.0 * K * nt + 2 * maps, flops=2 * fft + pt)
    ps, ss = _scales(c)
    prox = sum(_prox_flops(_dims(c), nt, p, s) for p, s in zip(ps, ss))
    ns = len(ps)
    # an iteration: gradient, the update (read g, x, u; write u, z), the prox (read z, write x)
    it = dict(bytes=(ns + 2) * image + maps + nvox * nt / 8 + (6 * ns + 1) * image, flops=2 * fft + pt + prox)
    f = 3.0 if kind == "grad" else 1.0   # the backward pass of an iteration does about twice its work
    return dict(bytes=f * c["niter"] * it["bytes"], flops=f * c["niter"] * it["flops"])


# --------------------------------------------------------------------------
# The same outputs in 64 bits
# --------------------------------------------------------------------------
def _svst64(X, beta):
    """U max(S - beta, 0) V^H of a batch (b, r, c), through the smaller Gram."""
    A = X if X.shape[-2] <= X.shape[-1] else X.mH
    lam, V = torch.linalg.eigh(A @ A.mH)
    s = lam.clamp_min(0).sqrt()
    h = torch.where(s > beta, (s - beta) / s.clamp_min(1e-300), torch.zeros_like(s))
    Y = (V * h[..., None, :]) @ (V.mH @ A)
    return Y if X.shape[-2] <= X.shape[-1] else Y.mH


def _prox64(img, beta, p, s):
    """patchSVST of (nt, nz, ny, nx) complex128: threshold every patch, average the overlaps."""
    nt, nz, ny, nx = img.shape
    px, py, pz = (min(a, b) for a, b in zip(p, (nx, ny, nz)))
    at = [(z, y, x) for z in _starts(nz, p[2], s[2]) for y in _starts(ny, p[1], s[1]) for x in _starts(nx, p[0], s[0])]
    out = torch.zeros_like(img)
    cnt = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    per = max(1, min(512, int(2e9 // (16 * nt * px * py * pz))))
    for b in range(0, len(at), per):
        P = torch.stack([img[:, z:z + pz, y:y + py, x:x + px].reshape(nt, -1) for z, y, x in at[b:b + per]])
        P = _svst64(P, beta)
        for (z, y, x), q in zip(at[b:b + per], P):
            out[:, z:z + pz, y:y + py, x:x + px] += q.reshape(nt, pz, py, px)
            cnt[z:z + pz, y:y + py, x:x + px] += 1
    return out / cnt.clamp_min(1)


def _normal64(X, maps, idx, ahy):
    """A'A of the summed scales minus A'y, frame by frame."""
    out = torch.empty_like(ahy)
    for t in range(X.shape[1]):
        out[t] = _adj(_fwd(X[:, t].to(C128).sum(0), maps, idx[t]), maps, idx[t]) - ahy[t]
    return out


def _adj_all64(y, maps, idx):
    return torch.stack([_adj(y[t].to(C128), maps, idx[t]) for t in range(y.shape[0])])


def _pogm64(ahy, maps, idx, ps, ss, lams, niter, L):
    """POGM with gradient restart as pogm_mod runs it with an in-place prox."""
    ns = len(ps)
    X = torch.zeros((ns,) + tuple(ahy.shape), dtype=C128, device=DEV)
    X[0] = ahy
    U, told, sig, flags = X.clone(), 1.0, 1.0, [False]
    for it in range(1, niter + 1):
        g = _normal64(X, maps, idx, ahy)
        a = 1 / L
        tnew = 0.5 * (1 + math.sqrt(1 + (8 if it == niter else 4) * told ** 2))
        b, c = (told - 1) / tnew, sig * told / tnew
        zeta = a * (1 + b + c)
        dot = n1 = n2 = 0.0
        for k in range(ns):
            u = X[k] - a * g
            d = u - U[k]
            yd = d if it > 1 else u - X[k]
            dot -= float((g * yd).real.sum())   # without conjugation, as the reference writes it
            Z = u + b * d + c * (u - X[k])
            U[k] = u
            X[k] = _prox64(Z, zeta * lams[k], ps[k], ss[k])
        restart = dot <= 0.0
        flags.append(restart)
        told = 1.0 if restart else tnew
    return X, flags


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "svst":
        X = _stack(c, seed)
        out = _svst64(X.to(C128), _threshold(c["keep"], c["m"], c["n"]))
        return out[0].t().contiguous() if c["batch"] == 1 else out
    if kind in ("patchsvst", "prox"):
        img = _series(_gen(seed), c["nt"], math.prod(_dims(c))).reshape(c["nt"], c["nz"], c["ny"], c["nx"])
        beta = _threshold(c["keep"], c["p"] ** 3, c["nt"])
        return _prox64(img.to(C128), beta, [c["p"]] * 3, [c["s"]] * 3)
    if kind in ("recon", "grad"):
        # eigenpairs in 64 bits take most of it: the large and the long ones are left out
        nvox = math.prod(_dims(c))
        if nvox * c["nt"] * c["niter"] * (1 if kind == "recon" else 2) > 8e7:
            return None
    maps, idx, y, x = _acquisition(c, seed)
    m64 = maps.to(C128)
    if kind == "sense":
        return {"y": torch.stack([_fwd(x[t].to(C128), m64, idx[t]) for t in range(c["nt"])]),
                "x": _adj_all64(y, m64, idx)}
    ahy = _adj_all64(y, m64, idx)
    if kind == "normal":
        X = torch.stack([x / c["ns"]] * c["ns"])
        X[0].mul_(0.9)
        return _normal64(X, m64, idx, ahy)
    ps, ss = _scales(c)
    nx, ny, nz = _dims(c)
    lams = [math.sqrt(math.prod(p)) + math.sqrt(c["nt"]) +
            math.sqrt(math.log(nx * ny * nz * c["nt"] / max(math.prod(p), c["nt"]))) for p in ps]
    X, flags = _pogm64(ahy, m64, idx, ps, ss, lams, c["niter"], float(len(ps)))
    if kind == "recon":
        return {"X": X, "restarts": flags}
    loss = 0.5 * float((X.sum(0) - x.to(C128)).abs().square().sum())
    return {"loss": loss, "grad": [None] * len(ps), "X": X, "restarts": flags}
