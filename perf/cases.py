"""Measured cases: the calls a user of this package makes, over their range.

A reconstruction uses three things: the projector and its transpose (alone,
under autograd, inside MLEM), the attenuation of the sample at every angle
(rotation, incident beam, detector cone), and the two whole schemes built on
them (the corrected MLEM with rebuilt attenuation, and the gradient through
it).  Sizes run from one 64^2 slice to 128^3 volumes at 120 angles and 256^2
slices at 180 angles, with odd sizes between.  All data are float32, as every
entry point takes it.  The inputs are made with plain torch from the seed
alone; `exact` repeats each pass with plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from fl_correction_b200.core import cal_atten_at_angles
from fl_correction_b200.cuda_lib import (backward_emission_batch, cal_atten_cuda, forward_emission,
                                         forward_emission_batch, forward_emission_batch_autograd,
                                         mlem_cuda, mlem_cuda_batch)
from fl_correction_b200.recon import CorrectedMLEM
from fl_correction_b200.xrf import XRFProjector


def listed():
    return [
        # one slice re-projected interactively: launch latency
        dict(name="project-slice", kind="project", A=60, B=1, H=64, W=64, R=1),
        # re-projection of a whole volume at every angle
        dict(name="project-volume", kind="project", A=120, B=128, H=128, W=128, R=1),
        # its transpose (sensitivities, custom update rules)
        dict(name="backproject-volume", kind="backproject", A=120, B=128, H=128, W=128, R=1),
        # training step of a network on the projector: forward and gradient, two
        # reference spectra, an odd slice size and count
        dict(name="autograd-refs", kind="autograd", A=75, B=33, H=101, W=101, R=2),
        # tuning on a single slice: many short dependent launches
        dict(name="mlem-slice", kind="mlem", A=90, B=1, H=96, W=96, R=1, n_iter=20, beta=1e-3),
        # one element of a volume between two attenuation rebuilds
        dict(name="mlem-volume", kind="mlem", A=120, B=128, H=128, W=128, R=1, n_iter=5, beta=1e-3),
        # slab of a large sample: slices of 256^2
        dict(name="mlem-large", kind="mlem", A=180, B=32, H=256, W=256, R=1, n_iter=2, beta=0.0),
        # fluorescence path sum of four lines at one angle
        dict(name="cone", kind="cone", K=4, Z=128, N=128, deg=13.3),
        # attenuation maps of two elements in a matrix, odd sizes
        dict(name="maps-ragged", kind="maps", L=2, S=61, N=111, A=40, deg=16.0, incident="own"),
        # the corrected MLEM: one rebuild and five iterations of three elements
        dict(name="corrected", kind="corrected", L=3, S=128, N=128, A=120, deg=13.3, n_iter=5,
             every=5),
        # gradient step through the attenuation
        dict(name="gradient", kind="gradient", L=3, S=96, N=96, A=90, deg=13.3),
        # the same for a slab of 256^2 slices, one chunk of angles, four elements
        dict(name="gradient-large", kind="gradient", L=4, S=64, N=256, A=8, deg=13.3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _samples(case):
    """Samples that one pass of the case visits (angles x voxels x passes)."""
    if case["kind"] == "cone":
        return case["K"] * case["Z"] * case["N"] ** 2 * 8
    if "L" in case:
        v = case["L"] * case["A"] * case["S"] * case["N"] ** 2
        return v * {"maps": 6, "corrected": 16 * case.get("n_iter", 0), "gradient": 24}[case["kind"]]
    v = case["R"] * case["A"] * case["B"] * case["H"] * case["W"]
    return v * {"project": 1, "backproject": 3, "autograd": 4}.get(case["kind"],
                                                                   4 * case.get("n_iter", 0) + 3)


def draw(rng):
    cap = 0.5 * max(_samples(c) for c in listed())
    while True:
        kind = rng.choice(["project", "backproject", "autograd", "mlem", "mlem", "cone", "maps",
                           "corrected", "gradient"])
        N = _log(rng, 48, 256)
        if kind == "cone":
            case = dict(kind=kind, K=rng.randint(1, 4), Z=_log(rng, 16, 192), N=min(N, 192),
                        deg=round(rng.uniform(9.0, 20.0), 1))
        elif kind in ("maps", "corrected", "gradient"):
            case = dict(kind=kind, L=rng.randint(1, 4), S=_log(rng, 16, 128), N=N,
                        A=_log(rng, 6, 90), deg=round(rng.uniform(9.0, 20.0), 1))
            if kind == "maps":
                case["incident"] = rng.choice(["own", "all"])
            if kind == "corrected":
                case.update(L=min(case["L"], 3), n_iter=rng.randint(2, 6), every=3)
        else:
            case = dict(kind=kind, A=_log(rng, 30, 180), B=_log(rng, 1, 160), H=N, W=N,
                        R=rng.choice([1, 1, 1, 2, 3]))
            if rng.random() < 0.15:
                case["W"] = _log(rng, 48, 256)
            if kind == "mlem":
                case.update(n_iter=rng.randint(1, 8), beta=rng.choice([0.0, 1e-3]))
        if _samples(case) <= cap:
            return case


def work(case):
    k = case["kind"]
    if k == "cone":
        vox = case["K"] * case["Z"] * case["N"] ** 2
        return {"bytes": 8 * vox, "flops": 2 * vox * 60}
    if "L" in case:
        L, A, vol = case["L"], case["A"], case["S"] * case["N"] ** 2
        vox = L * A * vol
        prj = L * A * case["S"] * case["N"]
        if k == "maps":          # fractions in, attenuation out
            return {"bytes": 4 * ((L + 1) * vol + vox), "flops": vox * 150}
        if k == "corrected":     # attenuation written per rebuild, read twice per iteration
            n, r = case["n_iter"], -(-case["n_iter"] // case["every"])
            return {"bytes": 4 * (vox * (r + r + 2 * n) + n * (2 * prj + 3 * L * vol)),
                    "flops": vox * (150 * r + 40 * n)}
        # nothing of size angles x volume has to leave the chip: C and the
        # projections in, projections and gradient out
        return {"bytes": 4 * (2 * L * vol + 2 * prj), "flops": vox * 600}
    A, B, H, W, R = (case[n] for n in ("A", "B", "H", "W", "R"))
    att, img, prj = A * B * H * W, R * B * H * W, A * B * W
    if k in ("project", "backproject"):
        return {"bytes": 4 * (att + img + prj), "flops": att * (2 + 8 * R)}
    if k == "autograd":
        return {"bytes": 4 * (2 * att + 2 * img + 2 * prj), "flops": att * (4 + 16 * R)}
    n = case["n_iter"]
    return {"bytes": 4 * (att * (2 * n + 1) + n * (2 * prj + 3 * img)),
            "flops": att * (2 + 8 * R) * (2 * n + 1)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed))


def _angles(A):
    """A projection angles over half a turn, in degrees."""
    return np.arange(A) * (180.0 / A)


def _theta(A, dev):
    return torch.tensor(_angles(A) / 180.0 * np.pi, dtype=torch.float32, device=dev)


def _grains(n, S, H, W, gen, dev):
    """(n, S, H, W) concentrations in [0, 0.9]: Voronoi grains of constant
    composition, summing to at most 0.9."""
    ns = 24
    seeds = torch.rand(ns, 3, generator=gen, device=dev)
    comp = torch.rand(ns, n, generator=gen, device=dev)
    z = torch.linspace(0, 1, S, device=dev)[:, None, None]
    y = torch.linspace(0, 1, H, device=dev)[None, :, None]
    x = torch.linspace(0, 1, W, device=dev)[None, None, :]
    best = torch.full((S, H, W), 9.0, device=dev)
    lab = torch.zeros((S, H, W), dtype=torch.long, device=dev)
    for k in range(ns):
        d = (z - seeds[k, 0]) ** 2 + (y - seeds[k, 1]) ** 2 + (x - seeds[k, 2]) ** 2
        lab = torch.where(d < best, k, lab)
        best = torch.minimum(best, d)
    comp = comp * (0.9 / float(comp.sum(1).max()))
    return comp.t()[:, lab].contiguous()


def _cone_mask(N, deg):
    """(M, N, M) acceptance of a round detector of full opening `deg` degrees
    seen from a voxel, per depth plane: the covered share of each cell along
    either axis, the plane's weights summing to the mean obliquity."""
    t = math.tan(math.radians(deg) / 2)
    m = int(math.ceil(N * t))
    k = np.abs(np.arange(-(m - 1), m))[:, None]
    d = np.arange(N)[None, :]
    p = np.clip(d * t + 0.5 - k, 0.0, 1.0) * np.sqrt(1.0 + (np.minimum(k, d * t) / np.maximum(d, 1)) ** 2)
    p[:, 0] = 0.0
    u = p / np.sqrt(np.maximum(p.sum(0), 1e-30))[None, :]
    return np.ascontiguousarray(u[:, :, None] * np.moveaxis(u[:, :, None], (0, 2), (2, 0)))


def _params(L, A, seed):
    """Reference-layout parameter dict of L elements in a matrix."""
    r = np.random.default_rng(seed)
    elems = ["Ca", "Fe", "Ni", "Zn"][:L]
    comps = [e + "_c" for e in elems]
    cs = {"elem_type": elems, "elem_compound": comps + ["matrix"]}
    rho = {c: float(r.uniform(2.5, 6.5)) for c in comps}
    rho["matrix"] = 1.0
    for c in comps:
        cs[c + "-x"] = np.full(A, r.uniform(25.0, 60.0))
        for e in elems:
            cs[c + "-" + e] = float(r.uniform(30.0, 60.0))
    cs["matrix-x"] = np.full(A, 5.0)
    for e in elems:
        cs["matrix-" + e] = 5.0
    return {"cs": cs, "rho": rho, "pix": 1e-4, "elem_type": elems, "elem_compound": comps + ["matrix"],
            "em_cs": {e: np.full(A, r.uniform(35.0, 42.0)) for e in elems}}


def _tables(param, A):
    """(A, n_ch) incident and (A, L, n_ch) fluorescence coefficients, (L, A)
    emission, in float64 of the float32 values that the call is given."""
    cs, rho, pix = param["cs"], param["rho"], param["pix"]
    comps, elems = param["elem_compound"], param["elem_type"]
    cx = np.array([[cs[c + "-x"][a] * rho[c] * pix for c in comps] for a in range(A)], np.float32)
    cf = np.array([[cs[c + "-" + e] * rho[c] * pix for c in comps] for e in elems], np.float32)
    em = np.array([param["em_cs"][e] * rho[c] * pix for e, c in zip(elems, comps)], np.float32)
    return cx.astype(np.float64), cf.astype(np.float64), em.astype(np.float64)


def _inputs(case, seed):
    """The tensors that the call takes, and nothing of this package."""
    dev = torch.device("cuda")
    gen = _gen(seed, dev)
    k = case["kind"]
    if k == "cone":
        mu = _grains(case["K"], case["Z"], case["N"], case["N"], gen, dev) * 0.03
        mask = torch.tensor(_cone_mask(case["N"], case["deg"]), dtype=torch.float32, device=dev)
        return dict(mu=mu.contiguous(), mask=mask)
    if "L" in case:
        L, S, N, A = (case[n] for n in ("L", "S", "N", "A"))
        frac = torch.cat([_grains(L, S, N, N, gen, dev), torch.ones((1, S, N, N), device=dev)])
        d = dict(frac=frac, param=_params(L, A, seed), mask=_cone_mask(N, case["deg"]))
        if k == "gradient":
            # residual of a fit under way: signed, smooth along the detector
            g = torch.randn((L, A, S, N), generator=gen, device=dev) * 0.05
            d["g"] = g.contiguous()
        if k == "corrected":
            em = _tables(d["param"], A)[2]
            th = _theta(A, dev)
            fall = torch.exp(-1e-2 * (torch.arange(N - 1, -1, -1, device=dev)[:, None]
                                      + 0.5 * torch.arange(N - 1, -1, -1, device=dev)[None, :]))
            I = torch.stack([torch.stack([_project(fall.expand(S, N, N), frac[l:l + 1], [em[l, a]],
                                                   th[a]) for a in range(A)]) for l in range(L)])
            I = I * (1.0 + 0.01 * torch.randn(I.shape, generator=gen, device=dev)).clamp_min(0.5)
            d["I"] = I.to(torch.float32).contiguous()
        return d
    A, B, H, W, R = (case[n] for n in ("A", "B", "H", "W", "R"))
    C = _grains(R, B, H, W, gen, dev)
    # beam from the far rows, detector beyond the last column, 10% structure
    ka, kb = 0.5 + 1.5 * torch.rand((2, A, 1, 1, 1), generator=gen, device=dev)
    h = torch.linspace(1, 0, H, device=dev)[:, None]
    w = torch.linspace(1, 0, W, device=dev)[None, :]
    atten = torch.rand((A, B, H, W), generator=gen, device=dev).mul_(-0.1).add_(1.0)
    atten.mul_(torch.exp(-ka * h - kb * w))
    em = 0.02 + 0.02 * torch.rand((A, R), generator=gen, device=dev)
    d = dict(C=C, atten=atten, em=em, theta=_theta(A, dev))
    if k in ("backproject", "autograd"):
        d["g"] = 0.5 + torch.rand((A, B, W), generator=gen, device=dev)
        if k == "autograd":
            d["g"] -= 1.0
    if k == "mlem":
        I = torch.stack([_project(atten[a], C, em[a].tolist(), d["theta"][a]) for a in range(A)])
        I = I * (1.0 + 0.01 * torch.randn(I.shape, generator=gen, device=dev)).clamp_min(0.5)
        d["I"] = I.to(torch.float32).contiguous()
        d["C"] = torch.ones_like(C)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    k = case["kind"]
    st = dict(d, case=case)
    if k == "project" and case["B"] == 1:       # the single-slice form
        st["atten"], st["C"] = d["atten"][:, 0].contiguous(), d["C"][:, 0].contiguous()
    if k == "mlem" and case["B"] == 1:
        st["atten"], st["C"] = d["atten"][:, 0].contiguous(), d["C"][:, 0].contiguous()
        st["I"] = d["I"][:, 0].contiguous()
    if k == "corrected":
        st["solver"] = CorrectedMLEM(d["param"], _angles(case["A"]), d["mask"],
                                     (case["S"], case["N"], case["N"]),
                                     fixed_frac=d["frac"][case["L"]:].cpu().numpy())
    if k == "gradient":
        st["proj"] = XRFProjector(d["param"], _angles(case["A"]), d["mask"],
                                  (case["S"], case["N"], case["N"]),
                                  fixed_frac=d["frac"][case["L"]:].cpu().numpy())
        st["C"] = d["frac"][:case["L"]].clone()
    if k == "autograd":
        st["C"] = d["C"].clone()
    return st


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "project":
        fn = forward_emission if case["B"] == 1 else forward_emission_batch
        return fn(s["atten"], s["C"], s["em"], s["theta"])
    if k == "backproject":
        return backward_emission_batch(s["atten"], s["g"], s["em"], s["theta"])
    if k == "autograd":
        C = s["C"].detach().requires_grad_(True)
        Pf = forward_emission_batch_autograd(s["atten"], C, s["em"], s["theta"])
        Pf.backward(s["g"])
        return Pf.detach(), C.grad
    if k == "mlem":
        fn = mlem_cuda if case["B"] == 1 else mlem_cuda_batch
        return fn(s["C"], s["atten"], s["em"], s["theta"], s["I"], case["n_iter"], case["beta"])
    if k == "cone":
        return cal_atten_cuda(s["mu"], s["mask"])
    if k == "maps":
        return cal_atten_at_angles(s["frac"], s["param"], _angles(case["A"]), s["mask"],
                                   incident=case["incident"])
    if k == "corrected":
        return s["solver"].run(s["I"], n_iter=case["n_iter"], recompute_every=case["every"])
    C = s["C"].detach().requires_grad_(True)
    Pf = s["proj"](C)
    Pf.backward(s["g"])
    return Pf.detach(), C.grad


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _taps(H, W, theta, dev):
    """Flat index of the low tap and the two bilinear fractions of every
    sample (h, w): rotation about the centre, clamped to the slice."""
    th = float(theta)
    c, s = math.cos(-th), math.sin(-th)
    cx, cy = (W - 1) / 2.0, (H - 1) / 2.0
    h = torch.arange(H, dtype=torch.float64, device=dev)[:, None] - cy
    w = torch.arange(W, dtype=torch.float64, device=dev)[None, :] - cx
    x = (c * h - s * w + cy).clamp(0, H - 1.001)
    y = (s * h + c * w + cx).clamp(0, W - 1.001)
    i0, j0 = torch.floor(x), torch.floor(y)
    return (i0.long() * W + j0.long()).reshape(-1), (x - i0).reshape(-1), (y - j0).reshape(-1)


def _weights(H, W, theta, dev, dtype):
    i, fx, fy = _taps(H, W, theta, dev)
    fx, fy = fx.to(dtype), fy.to(dtype)
    return ((i, (1 - fx) * (1 - fy)), (i + 1, (1 - fx) * fy), (i + W, fx * (1 - fy)),
            (i + W + 1, fx * fy))


def _project(att, C, em, theta):
    """att (B, H, W), C (R, B, H, W), em (R) -> (B, W), in C's type."""
    R, B, H, W = C.shape
    mix = sum(float(em[r]) * C[r] for r in range(R)).reshape(B, H * W)
    val = sum(mix[:, i] * w for i, w in _weights(H, W, theta, C.device, C.dtype))
    return (att.to(C.dtype) * val.reshape(B, H, W)).sum(dim=1)


def _backproject(out, att, g, em, theta):
    """out (R, B, H*W) += transpose of _project applied to g (B, W)."""
    B, H, W = att.shape
    q = (att.double() * g.double()[:, None, :]).reshape(B, H * W)
    one = torch.zeros((B, H * W), dtype=torch.float64, device=att.device)
    for i, w in _weights(H, W, theta, att.device, torch.float64):
        one.index_add_(1, i, q * w)
    for r in range(out.shape[0]):
        out[r] += float(em[r]) * one


def _mlem(C, atten, em, theta, I, n_iter, beta, delta=0.01):
    """C (R, B, H, W) double; atten (A, B, H, W); em (A, R)."""
    R, B, H, W = C.shape
    A = atten.shape[0]
    zero = lambda: torch.zeros((R, B, H * W), dtype=torch.float64, device=C.device)
    sens = zero()
    one = torch.ones((B, W), dtype=torch.float64, device=C.device)
    for a in range(A):
        _backproject(sens, atten[a], one, em[a], theta[a])
    sens = sens.clamp_min(1e-6).reshape(C.shape)
    for _ in range(n_iter):
        back = zero()
        for a in range(A):
            Pf = _project(atten[a], C, em[a], theta[a]).clamp_min(1e-6)
            _backproject(back, atten[a], I[a].double() / Pf, em[a], theta[a])
        den = sens
        if beta > 0:
            hub = torch.zeros_like(C)
            d = (C[..., 1:, :] - C[..., :-1, :]).clamp(-delta, delta)
            hub[..., 1:, :] += d
            hub[..., :-1, :] -= d
            d = (C[..., :, 1:] - C[..., :, :-1]).clamp(-delta, delta)
            hub[..., :, 1:] += d
            hub[..., :, :-1] -= d
            den = sens + beta * hub
        C = (C * back.reshape(C.shape) / den).clamp_min(0)
    return C


class _Cone(torch.autograd.Function):
    """res[k,z,x,y] = sum mask[dz,dx,dy] mu[k, z+dz-Mz//2, x+dx, y+dy-My//2] by
    the convolution theorem in (z, y), in 64 bits; linear, so its gradient is
    the same sum with the taps turned round."""

    @staticmethod
    def forward(ctx, mu, mask):
        ctx.mask = mask
        return _Cone.sum(mu, mask, False)

    @staticmethod
    def backward(ctx, g):
        return _Cone.sum(g.contiguous(), ctx.mask, True), None

    @staticmethod
    def sum(mu, mask, turned):
        K, Z, X, Y = mu.shape
        Mz, Mx, My = mask.shape
        Nz, Ny = Z + Mz, Y + My
        P = torch.fft.rfft2(mu.permute(0, 2, 1, 3), s=(Nz, Ny))         # (K, X, Nz, Nyh)
        m = torch.zeros((min(Mx, X), Nz, Ny), dtype=mu.dtype, device=mu.device)
        m[:, :Mz, :My] = mask.permute(1, 0, 2)[:X]
        m = torch.roll(m, (-(Mz // 2), -(My // 2)), (1, 2))
        G = torch.fft.rfft2(m)
        G = G if turned else G.conj()
        R = torch.zeros_like(P)
        for d in range(G.shape[0]):
            if turned:
                R[:, d:].addcmul_(P[:, :X - d], G[d])
            else:
                R[:, :X - d].addcmul_(P[:, d:], G[d])
        return torch.fft.irfft2(R, s=(Nz, Ny))[..., :Z, :Y].permute(0, 2, 1, 3).contiguous()


def _rotate(x, theta):
    """Bilinear rotation (n, S, N, N) about the centre, zero outside; the
    matrix entries are the float32 cosine and sine."""
    n, S, H, W = x.shape
    th = float(theta)
    c, s = float(np.float32(math.cos(th))), float(np.float32(math.sin(th)))
    cx = (W - 1) / 2.0
    h = torch.arange(H, dtype=torch.float64, device=x.device)[:, None] - cx
    w = torch.arange(W, dtype=torch.float64, device=x.device)[None, :] - cx
    px, py = c * w - s * h + cx, s * w + c * h + cx
    x0, y0 = torch.floor(px), torch.floor(py)
    flat = x.reshape(n * S, H * W)
    out = 0
    for dy in (0, 1):
        for dx in (0, 1):
            ix, iy = x0 + dx, y0 + dy
            wt = (1 - (px - ix).abs()) * (1 - (py - iy).abs())
            ok = (ix >= 0) & (ix < W) & (iy >= 0) & (iy < H)
            idx = (iy.clamp(0, H - 1) * W + ix.clamp(0, W - 1)).long().reshape(-1)
            out = out + flat[:, idx] * (wt * ok).reshape(-1)
    return out.reshape(n, S, H, W)


def _atten(frac, theta, cx, cf, mask, incident):
    """(L, S, N, N) attenuation at one angle: beam from the far rows, detector
    beyond the last column."""
    L = cf.shape[0]
    fr = _rotate(frac, theta)
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=frac.device)
    f = 1 - fr * t(cx)[:, None, None, None]
    f = f[:L] if incident == "own" else torch.prod(f, dim=0, keepdim=True).expand(L, -1, -1, -1)
    inc = torch.flip(torch.cumprod(torch.flip(f, [2]), dim=2), [2])
    inc = torch.cat([inc[:, :, 1:], torch.ones_like(inc[:, :, :1])], dim=2)
    mu = torch.einsum("ij,jshw->ishw", t(cf), fr)
    # the cone's frame: depth towards the detector, columns against the beam
    res = _Cone.apply(torch.flip(mu.transpose(2, 3), [3]).contiguous(), mask)
    return inc * torch.exp(-torch.flip(res, [3]).transpose(2, 3))


def exact(case, seed):
    d = _inputs(case, seed)
    k = case["kind"]
    D = torch.float64
    if k == "cone":
        return _Cone.sum(d["mu"].to(D), d["mask"].to(D), False)
    if "L" not in case:
        A, B, H, W, R = (case[n] for n in ("A", "B", "H", "W", "R"))
        if k == "mlem":
            # about a second per 1e9 scattered taps
            if 4 * A * B * H * W * (case["n_iter"] + 1) > 1.2e10:
                return None
            C = _mlem(d["C"].to(D), d["atten"], d["em"].to(D), d["theta"], d["I"], case["n_iter"],
                      case["beta"])
            return C[:, 0] if B == 1 else C
        Pf = C = None
        if k != "backproject":
            Pf = torch.stack([_project(d["atten"][a], d["C"].to(D), d["em"][a].to(D), d["theta"][a])
                              for a in range(A)])
        if k != "project":
            C = torch.zeros((R, B, H * W), dtype=D, device=d["C"].device)
            for a in range(A):
                _backproject(C, d["atten"][a], d["g"][a], d["em"][a].to(D), d["theta"][a])
            C = C.reshape(R, B, H, W)
        if k == "project":
            return Pf[:, 0] if B == 1 else Pf
        return C if k == "backproject" else (Pf, C)
    L, A, N = case["L"], case["A"], case["N"]
    cx, cf, em = _tables(d["param"], A)
    theta = _theta(A, d["frac"].device)
    mask = torch.tensor(d["mask"], dtype=D, device=d["frac"].device)
    frac = d["frac"].to(D)
    if k == "maps":
        return torch.stack([_atten(frac, theta[a], cx[a], cf, mask, case["incident"])
                            for a in range(A)], dim=1)
    if k == "corrected":
        C = torch.ones_like(frac[:L])
        done = 0
        while done < case["n_iter"]:
            n = min(case["every"], case["n_iter"] - done)
            f = C.clamp(0, 1)
            f = torch.cat([f / f.sum(0, keepdim=True).clamp_min(1), frac[L:]])
            att = torch.stack([_atten(f, theta[a], cx[a], cf, mask, "own") for a in range(A)], dim=1)
            C = torch.cat([_mlem(C[l:l + 1], att[l], em[l][:, None], theta, d["I"][l], n, 0.0)
                           for l in range(L)])
            done += n
        return C
    grad = torch.zeros_like(frac[:L])
    Pf = []
    for a in range(A):
        C = frac[:L].clone().requires_grad_(True)
        att = _atten(torch.cat([C, frac[L:]]), theta[a], cx[a], cf, mask, "own")
        p = torch.stack([_project(att[l], C[l:l + 1], [em[l, a]], theta[a]) for l in range(L)])
        p.backward(d["g"][:, a].to(D))
        grad += C.grad
        Pf.append(p.detach())
    return torch.stack(Pf, dim=1), grad
