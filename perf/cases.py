"""Workloads whose time is followed from change to change: the calls that a
reconstruction makes, one layer at a time, through the package's public entry
points, over the sizes that its configurations use.

A reconstruction slices a model at reference orientations, matches frames to
the slices, merges the oriented frames (type-1 NUFFTs and a CG solve) and
phases the result; each of those calls is a kind here:

  slice     NUFFT.set_model + slice_real, FP32 (eps 1e-6) or FP64 (eps 1e-12)
  forward   autocorrelation.forward: type 2 at explicit points, complex
  adjoint   autocorrelation.adjoint: type 1 at explicit points
  match     FrameSet.from_counts + match_bf16 against resident references
  argmin32  argmin_fp32: the plain FP32 match of a batch of slices
  argmin64  argmin_fp64: the same at the reference's double precision
  merge     MergeOperator.cg, Toeplitz form
  phase     sequential.phasing.phase: the whole phase-retrieval call
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spinifel_gb300 import autocorrelation, geom, matching
from spinifel_gb300.extern.nufft_ext import NUFFT
from spinifel_gb300.merge import MergeOperator, antisupport
from spinifel_gb300.sequential.phasing import phase
from spinifel_gb300.settings import Settings

# 64-bit answers are direct sums; past this many FP64 operations they take too long
EXACT_FLOPS = 1.2e13


def listed():
    return [
        # one matching batch of the small configuration (41^3 model, 4 x 32 x 32
        # pixels): 100 orientations, the smallest call of the loop
        {"name": "slice_batch_41", "kind": "slice", "M": 41, "panels": 4, "nx": 32, "ny": 32,
         "n_orient": 100, "fp64": False, "bf16": False},
        # reference slices of the full-size configuration (81^3, 4 x 128 x 128
        # pixels) with the bf16 copy the tensor-core match reads
        {"name": "slice_refs_81", "kind": "slice", "M": 81, "panels": 4, "nx": 128, "ny": 128,
         "n_orient": 2000, "fp64": False, "bf16": True},
        # slices at the reference's own precision (eps 1e-12 in double)
        {"name": "slice_fp64_41", "kind": "slice", "M": 41, "panels": 4, "nx": 32, "ny": 32,
         "n_orient": 100, "fp64": True, "bf16": False},
        # forward operator at the pixels of 97 frames of a detector with odd sides
        {"name": "forward_61_ragged", "kind": "forward", "M": 61, "panels": 3, "nx": 50, "ny": 37,
         "n_orient": 97, "eps": 1e-6},
        # adjoint of the small configuration: 500 frames of 4,096 pixels
        {"name": "adjoint_41", "kind": "adjoint", "M": 41, "panels": 4, "nx": 32, "ny": 32,
         "n_orient": 500, "eps": 1e-6},
        # adjoint on the large merge grid: 200 frames of 65,536 pixels
        {"name": "adjoint_151", "kind": "adjoint", "M": 151, "panels": 4, "nx": 128, "ny": 128,
         "n_orient": 200, "eps": 1e-6},
        # one serving request of a few frames against resident references
        {"name": "match_request", "kind": "match", "M": 81, "panels": 4, "nx": 128, "ny": 128,
         "n_img": 5, "n_ref": 20000},
        # a large batch of frames against resident references
        {"name": "match_batch", "kind": "match", "M": 81, "panels": 4, "nx": 128, "ny": 128,
         "n_img": 4096, "n_ref": 50000},
        # plain FP32 match of one batch of slices, odd counts and an odd pixel number
        {"name": "argmin32_odd", "kind": "argmin32", "M": 41, "panels": 3, "nx": 50, "ny": 37,
         "n_img": 333, "n_ref": 1999},
        # the small configuration's match in double: 500 frames, 2,000 references
        {"name": "argmin64_41", "kind": "argmin64", "M": 41, "panels": 4, "nx": 32, "ny": 32,
         "n_img": 500, "n_ref": 2000},
        # merge solve at the full-size configuration's grid
        {"name": "merge_cg_81", "kind": "merge", "M": 81, "n_iter": 30},
        # phase retrieval with the default settings (M = 81)
        {"name": "phase_81", "kind": "phase", "Mquat": 20, "loops": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _detector(rng, most=128):
    return {"panels": rng.choice([1, 2, 3, 4, 4, 4]), "nx": _log(rng, 16, most),
            "ny": _log(rng, 16, most)}


def draw(rng):
    kind = rng.choice(["slice", "slice", "slice64", "forward", "adjoint", "adjoint", "match",
                       "match", "argmin32", "argmin64", "merge", "phase"])
    if kind in ("slice", "slice64"):
        d = _detector(rng)
        fp64 = kind == "slice64"
        pts = _log(rng, 2e4, 5e5) if fp64 else _log(rng, 5e4, 1e8)
        n = max(1, pts // (d["panels"] * d["nx"] * d["ny"]))
        return {"kind": "slice", "M": rng.randrange(21, 62 if fp64 else 100, 2), **d,
                "n_orient": n, "fp64": fp64,
                "bf16": not fp64 and (d["panels"] * d["nx"] * d["ny"]) % 8 == 0
                and rng.random() < 0.5}
    if kind in ("forward", "adjoint"):
        d = _detector(rng)
        pts = _log(rng, 5e4, 3e6 if kind == "forward" else 1e7)
        n = max(1, pts // (d["panels"] * d["nx"] * d["ny"]))
        return {"kind": kind, "M": rng.randrange(21, 152, 2), **d, "n_orient": n,
                "eps": rng.choice([1e-6, 1e-6, 1e-4])}
    if kind == "match":
        d = _detector(rng)
        return {"kind": kind, "M": 81, **d, "n_img": _log(rng, 1, 4000),
                "n_ref": _log(rng, 2000, 50000)}
    if kind in ("argmin32", "argmin64"):
        d = _detector(rng, 128 if kind == "argmin32" else 48)
        p = d["panels"] * d["nx"] * d["ny"]
        n_img, n_ref = _log(rng, 10, 1500), _log(rng, 100, 8000)
        cap = 1e11 if kind == "argmin32" else 4e9
        n_img = max(1, min(n_img, int(cap / (n_ref * p))))
        return {"kind": kind, "M": 41, **d, "n_img": n_img, "n_ref": n_ref}
    if kind == "merge":
        return {"kind": kind, "M": rng.randrange(31, 112, 2), "n_iter": rng.randrange(5, 31)}
    return {"kind": "phase", "Mquat": rng.randrange(5, 25), "loops": rng.randrange(1, 6)}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
DEV = "cuda"


def _blobs(M, rng, n_blobs=20):
    """A density of 20 Gaussian blobs in the inner half of the box (device FP64)."""
    ax = torch.arange(M, dtype=torch.float64, device=DEV) - M // 2
    rho = torch.zeros(M, M, M, dtype=torch.float64, device=DEV)
    for _ in range(n_blobs):
        c = rng.uniform(-M / 4, M / 4, 3)
        s, a = rng.uniform(1.0, 3.0), rng.uniform(0.5, 1.0)
        g = [torch.exp(-(ax - float(v)) ** 2 / (2 * s * s)) for v in c]
        rho += a * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
    return rho


def _intensity(M, rng):
    """|FFT(density)|^2, centred, largest value 1."""
    f = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(_blobs(M, rng))))
    i = f.real ** 2 + f.imag ** 2
    return i / i.max()


def _geometry(case):
    ppr, dist = geom.flat_detector(case["panels"], case["nx"], case["ny"])
    return ppr, dist


def _rotations(quats):
    q = torch.as_tensor(quats, dtype=torch.float64, device=DEV)
    w, x, y, z = q.unbind(1)
    r = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1)
    return r.reshape(-1, 3, 3).transpose(1, 2)  # the inverse rotation


def _points(case, rng, n_orient):
    """(H, K, L) in radians of every detector pixel at n_orient orientations: FP64."""
    ppr, dist = _geometry(case)
    mult = math.pi / float(dist.max())
    rinv = _rotations(geom.uniform_quaternions(n_orient, rng))
    p = torch.as_tensor(ppr.reshape(3, -1), dtype=torch.float64, device=DEV) * mult
    return torch.matmul(rinv, p).permute(1, 0, 2).reshape(3, -1)


def _patterns(case, vol, rng, n, out=None):
    """n diffraction patterns [n, n_pix]: the intensity volume sampled
    trilinearly at the rotated pixels, a beam stop over the centre, FP32."""
    ppr, dist = _geometry(case)
    n_pix = ppr[0].size
    p = torch.as_tensor(ppr.reshape(3, -1) / dist.max(), dtype=torch.float32, device=DEV)
    stop = 1 - torch.exp(-(p.square().sum(0) / 0.1 ** 2))
    rinv = _rotations(geom.uniform_quaternions(n, rng)).float()
    out = torch.empty(n, n_pix, dtype=torch.float32, device=DEV) if out is None else out
    step = max(1, (1 << 26) // n_pix)
    v = vol.float()[None, None]
    for st in range(0, n, step):
        q = torch.matmul(rinv[st:st + step], p)  # [b, 3, n_pix] in [-1, 1]
        g = q.flip(1).permute(0, 2, 1).reshape(1, 1, 1, -1, 3)  # sampled as (x, y, z)
        s = torch.nn.functional.grid_sample(v, g, mode="bilinear", align_corners=True)
        out[st:st + step] = s.reshape(-1, n_pix) * stop
    return out


def _match_inputs(case, seed, photons):
    """Frames (Poisson counts at `photons` a pixel) and reference slices of
    one volume at independent orientations, in the frames' scale."""
    rng = np.random.default_rng(seed)
    vol = _intensity(case["M"], rng)
    refs = _patterns(case, vol, rng, case["n_ref"])
    lam = _patterns(case, vol, rng, case["n_img"])
    scale = photons / float(refs[:256].double().mean())
    refs *= scale
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)
    counts = torch.empty(case["n_img"], refs.shape[1], dtype=torch.int16, device=DEV)
    for st in range(0, case["n_img"], 512):
        c = torch.poisson(lam[st:st + 512] * scale, generator=gen)
        counts[st:st + 512] = c.clamp_(max=32767).to(torch.int16)
    return counts, refs


def _merge_inputs(case, seed):
    """Toeplitz kernel of points spread evenly over orientations (its modes
    are the mean of sin(kq)/(kq) over the detector's radii), right-hand side
    of a blob density's autocorrelation with noise."""
    M = case["M"]
    mu = 2 * M
    rng = np.random.default_rng(seed)
    ppr, dist = geom.flat_detector(4, 32, 32)
    n_pts = 500 * dist.size
    q = torch.as_tensor(np.sort(dist.reshape(-1))[::8] * (math.pi / dist.max()), device=DEV)
    r2 = torch.arange(0, 3 * M * M + 1, dtype=torch.float64, device=DEV)
    table = torch.sinc(r2.sqrt()[:, None] * (q / math.pi)[None, :]).mean(1) * (n_pts / mu ** 3)
    d = torch.arange(mu, device=DEV) - M
    s = d * d
    conv = table[s[:, None, None] + s[None, :, None] + s[None, None, :]]
    rho = _blobs(M, rng)
    f = torch.fft.fftn(rho)
    ac = torch.fft.fftshift(torch.fft.ifftn(f.real ** 2 + f.imag ** 2).real)
    ac /= ac.max()
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 5)
    noise = torch.randn(ac.shape, dtype=torch.float64, device=DEV, generator=gen)
    b = _toeplitz(conv, ac) / M ** 3
    b += 1e-3 * b.std() * (noise + noise.flip(0, 1, 2))
    return conv, b.reshape(-1), 1.0 / n_pts / 1000.0, 1e3


def _toeplitz(conv, x):
    """sum_d conv[d + M] x[k - d] on the M^3 grid, |d| < M, in FP64."""
    M = x.shape[0]
    k = torch.fft.rfftn(torch.roll(conv, (-M, -M, -M), (0, 1, 2)))
    pad = torch.zeros_like(conv)
    pad[:M, :M, :M] = x
    return torch.fft.irfftn(torch.fft.rfftn(pad) * k, s=conv.shape)[:M, :M, :M]


def _phase_inputs(case, seed):
    M = 4 * case["Mquat"] + 1
    rng = np.random.default_rng(seed)
    rho = _blobs(M, rng)
    f = torch.fft.fftn(rho)
    ac = torch.fft.fftshift(torch.fft.ifftn(f.real ** 2 + f.imag ** 2).real)
    sup = torch.fft.ifftshift(rho) > 1e-2 * rho.max()
    start = torch.as_tensor(rng.random((M, M, M)), device=DEV) * sup
    return ac.cpu().numpy(), sup.cpu().numpy(), start.cpu().numpy()


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def _settings(case):
    return Settings(N_orientations=case.get("n_orient", 1), N_batch_size=case.get("n_orient", 1),
                    M_override=case["M"], use_single_prec=not case.get("fp64", False),
                    reduced_det_shape_override=(case["panels"], case["nx"], case["ny"]))


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    st = {"case": case}
    if kind == "slice":
        ppr, dist = _geometry(case)
        st["model"] = _intensity(case["M"], rng)
        st["nufft"] = NUFFT(_settings(case), ppr, dist,
                            ref_orientations=geom.uniform_quaternions(case["n_orient"], rng))
        n_pix = ppr[0].size
        dt = torch.float64 if case["fp64"] else torch.float32
        st["out"] = torch.empty(case["n_orient"], n_pix, dtype=dt, device=DEV)
        st["bf16"] = torch.empty(case["n_orient"], n_pix, dtype=torch.bfloat16, device=DEV) \
            if case["bf16"] else None
    elif kind in ("forward", "adjoint"):
        st["hkl"] = tuple(_points(case, rng, case["n_orient"]).float())
        n = st["hkl"][0].numel()
        if kind == "forward":
            st["model"] = _intensity(case["M"], rng)
        else:
            gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
            st["data"] = torch.poisson(torch.full((n,), 2.0, dtype=torch.float64, device=DEV),
                                       generator=gen)
    elif kind == "match":
        counts, refs = _match_inputs(case, seed, 0.5)
        st["counts"], st["refs"] = counts, matching.ReferenceSet(refs)
    elif kind in ("argmin32", "argmin64"):
        counts, refs = _match_inputs(case, seed, 2.0)
        dt = torch.float32 if kind == "argmin32" else torch.float64
        st["frames"], st["refs"] = counts.to(dt), refs.to(dt)
    elif kind == "merge":
        conv, st["b"], rl, fl = _merge_inputs(case, seed)
        M = case["M"]
        st["op"] = MergeOperator(M, 2 * M, rl, fl, torch.ones(M, M, M, device=DEV),
                                 antisupport(M, 1))
        st["op"].set_kernel(conv.float())
        st["x0"] = torch.zeros(M ** 3, dtype=torch.float64, device=DEV)
    else:
        st["ac"], st["sup"], st["rho"] = _phase_inputs(case, seed)
        st["settings"] = Settings(Mquat_override=case["Mquat"], N_phase_loops=case["loops"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "slice":
        plan = st["nufft"].set_model(st["model"])
        st["nufft"].slice_real(plan, 0, case["n_orient"], out=st["out"], out_bf16=st["bf16"])
        return [st["out"], st["bf16"]] if case["bf16"] else [st["out"]]
    if kind == "forward":
        h, k, l = st["hkl"]
        return [autocorrelation.forward(st["model"], h, k, l, 1, True, h.numel(),
                                        eps=case["eps"])]
    if kind == "adjoint":
        h, k, l = st["hkl"]
        return [autocorrelation.adjoint(st["data"], h, k, l, case["M"], eps=case["eps"])]
    if kind == "match":
        return list(matching.match_bf16(matching.FrameSet.from_counts(st["counts"]), st["refs"]))
    if kind == "argmin32":
        return list(matching.argmin_fp32(st["frames"], st["refs"]))
    if kind == "argmin64":
        return list(matching.argmin_fp64(st["frames"], st["refs"]))
    if kind == "merge":
        x, iters, _ = st["op"].cg(st["b"], st["x0"], case["n_iter"], history=False)
        return [x, iters]
    return list(phase(1, st["ac"], st["sup"], st["rho"], settings=st["settings"]))


def _n_pts(case):
    return case["n_orient"] * case["panels"] * case["nx"] * case["ny"]


def work(case):
    kind = case["kind"]
    if kind in ("slice", "forward", "adjoint"):
        # kernel width at the tolerance; 2 w^3 operations a point and part,
        # and the transform of the twice oversampled grid
        w = 13 if case.get("fp64") else round(-math.log10(case.get("eps", 1e-6))) + 1
        n, m3 = _n_pts(case), case["M"] ** 3
        fft = 5 * 8 * m3 * math.log2(8 * m3)
        parts = 2 if kind == "forward" else 1
        out = n * (8 if case.get("fp64") else 4) * parts + (n * 2 if case.get("bf16") else 0)
        if kind == "adjoint":
            return {"bytes": n * (12 + 8) + 4 * m3, "flops": n * 2 * w ** 3 + fft}
        inp = 8 * m3 + (n * 12 if kind == "forward" else 0)
        return {"bytes": out + inp, "flops": parts * n * 2 * w ** 3 + fft}
    if kind in ("match", "argmin32", "argmin64"):
        p = case["panels"] * case["nx"] * case["ny"]
        size = {"match": 2, "argmin32": 4, "argmin64": 8}[kind]
        frames = 2 if kind == "match" else size
        return {"bytes": p * (case["n_ref"] * size + case["n_img"] * frames),
                "flops": 2 * p * case["n_ref"] * case["n_img"]}
    if kind == "merge":
        m3 = case["M"] ** 3
        # each iteration: the transforms of the convolution (8 M^3, single) and
        # of the regulariser (M^3, double) there and back, and the vectors once
        it = 2 * 2.5 * 8 * m3 * math.log2(8 * m3) + 2 * 2.5 * m3 * math.log2(m3) + 20 * m3
        return {"bytes": case["n_iter"] * m3 * 8 * 9, "flops": case["n_iter"] * it}
    m3 = (4 * case["Mquat"] + 1) ** 3
    its = case["loops"] * 25 + 10
    return {"bytes": its * m3 * 80, "flops": its * 2 * 2.5 * m3 * math.log2(m3)}


# ---------------------------------------------------------------------------
# the same answers in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _phases(x, M):
    k = torch.arange(M, dtype=torch.float64, device=DEV) - M // 2
    a = x[:, None] * k[None, :]
    return torch.cos(a), torch.sin(a)


def _direct_t2(f, x, y, z):
    """sum_k f_k exp(-i k.x) at every point (f real)."""
    m1, m2, m3 = f.shape
    re, im = torch.empty_like(x), torch.empty_like(x)
    step = max(1, (1 << 28) // (m1 * m2 * 2))
    for st in range(0, x.numel(), step):
        s = slice(st, st + step)
        c3, s3 = _phases(z[s], m3)
        tr = torch.matmul(f.reshape(-1, m3), c3.T).reshape(m1, m2, -1)
        ti = -torch.matmul(f.reshape(-1, m3), s3.T).reshape(m1, m2, -1)
        c2, s2 = _phases(y[s], m2)
        ur = (torch.einsum("abp,pb->ap", tr, c2) + torch.einsum("abp,pb->ap", ti, s2))
        ui = (torch.einsum("abp,pb->ap", ti, c2) - torch.einsum("abp,pb->ap", tr, s2))
        c1, s1 = _phases(x[s], m1)
        re[s] = (ur.T * c1 + ui.T * s1).sum(1)
        im[s] = (ui.T * c1 - ur.T * s1).sum(1)
    return re, im


def _direct_t1(c, x, y, z, M):
    """Re sum_j c_j exp(i k.x_j) on the M^3 modes (c real)."""
    out = torch.zeros(M * M, M, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 27) // (M * M))
    for st in range(0, x.numel(), step):
        s = slice(st, st + step)
        c1, s1 = _phases(x[s], M)
        c2, s2 = _phases(y[s], M)
        c3, s3 = _phases(z[s], M)
        c1, s1 = c1 * c[s, None], s1 * c[s, None]
        er = c1[:, :, None] * c2[:, None, :] - s1[:, :, None] * s2[:, None, :]
        ei = c1[:, :, None] * s2[:, None, :] + s1[:, :, None] * c2[:, None, :]
        out += torch.matmul(er.reshape(er.shape[0], -1).T, c3)
        out -= torch.matmul(ei.reshape(ei.shape[0], -1).T, s3)
    return out.reshape(M, M, M)


def _exact_match(frames, refs, per=512):
    """Smallest distance of every frame in FP64, over the nearest 16 in FP32."""
    out = torch.empty(frames.shape[0], dtype=torch.float64, device=DEV)
    sq = torch.cat([r.double().square().sum(1) for r in refs.split(1024)])
    for st in range(0, frames.shape[0], per):
        x = frames[st:st + per]
        d = sq[None, :].float() - 2 * torch.matmul(x.float(), refs.float().T)
        near = d.topk(min(16, refs.shape[0]), largest=False).indices
        for i in range(x.shape[0]):
            out[st + i] = (refs[near[i]].double() - x[i].double()).square().sum(1).min()
    return out


def _exact_cg(conv, b, rl, fl, M, n_iter, rtol=1e-5):
    lu = np.linspace(-math.pi, math.pi, M)
    g = np.meshgrid(lu, lu, lu, indexing="ij")
    anti = torch.as_tensor(np.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2) > math.pi, device=DEV)
    mask = torch.fft.ifftshift(anti.double())
    kern = torch.fft.rfftn(torch.roll(conv, (-M, -M, -M), (0, 1, 2)))
    pad = torch.zeros_like(conv)

    def op(v):
        x = v.reshape(M, M, M)
        pad[:M, :M, :M] = x
        t = torch.fft.irfftn(torch.fft.rfftn(pad) * kern, s=conv.shape)[:M, :M, :M] / M ** 3
        r = torch.fft.fftshift(torch.fft.ifftn(torch.fft.fftn(torch.fft.ifftshift(x))
                                               * mask).real)
        return (t + rl * x + fl * r).reshape(-1)

    x, r, p, rho0 = torch.zeros_like(b), b.clone(), None, 1.0
    atol = rtol * float(b.norm())
    for _ in range(n_iter):
        rho = float(torch.dot(r, r))
        if math.sqrt(rho) < atol:
            break
        p = r.clone() if p is None else r + (rho / rho0) * p
        q = op(p)
        a = rho / float(torch.dot(p, q))
        x += a * p
        r -= a * q
        rho0 = rho
    return x


def _gauss(x, wrap):
    """gaussian_filter with sigma 1 cut at 2 sigma, periodic or zero outside."""
    w = np.exp(-0.5 * np.arange(-2, 3) ** 2)
    w = w / w.sum()
    for ax in range(3):
        acc = x * w[2]
        for j in (1, 2):
            lo, hi = torch.roll(x, j, ax), torch.roll(x, -j, ax)
            if not wrap:
                lo.narrow(ax, 0, j).zero_()
                hi.narrow(ax, x.shape[ax] - j, j).zero_()
            acc = acc + (lo + hi) * w[2 + j]
        x = acc
    return x


def _exact_phase(ac, sup, rho, loops, n_er=10, n_hio=5, beta=0.9):
    M = ac.shape[0]
    ac, sup, rho = (torch.as_tensor(a, device=DEV) for a in (ac, sup, rho))
    amp = torch.fft.fftn(torch.fft.ifftshift(_gauss(ac.clamp(min=0), False))).abs().sqrt()

    def project(r):
        f = torch.fft.fftn(r)
        g = torch.polar(amp, f.angle())
        g[0, 0, 0] = f[0, 0, 0]
        return torch.fft.ifftn(g).real

    def er(r, n):
        for _ in range(n):
            m = project(r)
            r = torch.where(sup & (m > 0), m, torch.zeros_like(m))
        return r

    for _ in range(loops):
        rho = er(rho, n_er)
        for _ in range(n_hio):
            m = project(rho)
            rho = torch.where(sup & (m > 0), m, rho - beta * m)
        rho = er(rho, n_er)
        g = _gauss(rho.abs(), True)
        sup = g > g.std(unbiased=False)
    rho = er(rho, n_er)
    c = torch.as_tensor(np.linspace(-1, 1, M + 1), device=DEV)
    c = torch.fft.ifftshift((c[:-1] + c[1:]) / 2)
    a = rho.abs()
    shift = []
    for ax in range(3):
        v = [None, None, None]
        v[ax] = slice(None)
        shift.append(int(np.round(float((a * c[tuple(v)]).sum() / a.sum()) * M / 2)))
    rho = torch.roll(rho, [-s for s in shift], (0, 1, 2))
    f = torch.fft.fftn(rho).abs() ** 2
    return torch.fft.fftshift(torch.fft.ifftn(f).abs()), rho


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("slice", "forward", "adjoint"):
        if 4.0 * case["M"] ** 3 * _n_pts(case) > EXACT_FLOPS:
            return None
    if kind == "slice":
        model = _intensity(case["M"], rng)
        if not case["fp64"]:
            model = model.float().double()
        x, y, z = _points(case, rng, case["n_orient"])
        re = _direct_t2(model, x, y, z)[0].reshape(case["n_orient"], -1)
        return [re, re] if case["bf16"] else [re]
    if kind in ("forward", "adjoint"):
        x, y, z = _points(case, rng, case["n_orient"]).float().double()
        if kind == "forward":
            return [torch.complex(*_direct_t2(_intensity(case["M"], rng), x, y, z))]
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
        c = torch.poisson(torch.full_like(x, 2.0), generator=gen)
        return [_direct_t1(c, x, y, z, case["M"]) / case["M"] ** 3]
    if kind in ("match", "argmin32", "argmin64"):
        counts, refs = _match_inputs(case, seed, 0.5 if kind == "match" else 2.0)
        return [None, _exact_match(counts.float(), refs)]
    if kind == "merge":
        conv, b, rl, fl = _merge_inputs(case, seed)
        return [_exact_cg(conv, b, rl, fl, case["M"], case["n_iter"]), None]
    ac, sup, rho = _phase_inputs(case, seed)
    a, r = _exact_phase(ac, sup, rho, case["loops"])
    return [a, None, r]
