"""Cases that say how fast the framework does the work its users have it do.

The path is the one the drivers walk: raw projections -> sinograms (`prep`), sinograms -> images (`fbp`),
images -> sinograms (`radon`), total-variation reconstruction of one slice, of a batch of slices and of a
ragged batch of problems (`tv`, `ragged`), and the registration-aware objective with both of its gradients
(`grad`).  Everything goes through the package's public classes; device arrays are torch tensors, except for the
ragged batch, whose entry point takes host arrays.

`exact` evaluates the same formulas in double precision with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from acumen_gb300.batch import RaggedBatch
from acumen_gb300.preprocess import Preprocessor
from acumen_gb300.tomography import Tomography

DEV = "cuda"
LAM, MU, EPS = 0.05, 1.0, 0.05   # the regularisation every configuration of the framework uses
I0 = 5e3                         # counts per detector bin behind the synthetic sinograms


# ---- the cases -----------------------------------------------------------------------------------------------------

def listed():
    return [
        # one small slice, looked at interactively: latency and launches
        {"name": "fbp_129", "kind": "fbp", "N": 129, "T": 90, "S": 1, "closed": False},
        # one slice of plain FBP at the 725-bin, 720-angle configuration
        {"name": "fbp_725", "kind": "fbp", "N": 725, "T": 720, "S": 1, "closed": False},
        # FBP of a whole stack: 256 slices of 2048 detector bins at 1200 angles, the warm start of the big solve
        {"name": "fbp_2049x256", "kind": "fbp", "N": 2049, "T": 1200, "S": 256, "closed": True},
        # forward projection of one slice at the single-slice TV configuration (1449 bins, 900 angles)
        {"name": "radon_1449", "kind": "radon", "N": 1449, "T": 900, "S": 1, "closed": False},
        # a batch that fills no group evenly, odd angle count
        {"name": "radon_1025x37", "kind": "radon", "N": 1025, "T": 601, "S": 37, "closed": True},
        # forward projection of the whole stack, the operator the big solve spends most of its time in
        {"name": "radon_2049x256", "kind": "radon", "N": 2049, "T": 1200, "S": 256, "closed": True},
        # split-Bregman TV of one slice (1449 bins, 900 angles): warm start, one outer iteration, a few CG steps
        {"name": "tv_1449", "kind": "tv", "N": 1449, "T": 900, "S": 1, "nouter": 1, "ncg": 3, "closed": False},
        # the same for a batch of slices of a 1024-bin detector
        {"name": "tv_1025x64", "kind": "tv", "N": 1025, "T": 600, "S": 64, "nouter": 1, "ncg": 3, "closed": True},
        # independent problems of uneven side and angle count, solved together from host arrays
        {"name": "ragged_6", "kind": "ragged", "P": 6, "Nmax": 1449, "Tmax": 900, "nouter": 1, "ncg": 3},
        # loss and gradients with respect to the image and the per-angle detector offsets
        {"name": "grad_1025x2", "kind": "grad", "N": 1025, "T": 750, "S": 2},
        # counts -> normalised projections -> axis by cross-correlation -> median, resample, sinograms
        {"name": "prep_2048x256", "kind": "prep", "D": 2048, "R": 256, "P": 180, "mode": 1, "reg": "xcorr"},
        # the same for a small odd detector with the axis found by the pattern search (the drivers' default)
        {"name": "prep_1025x64", "kind": "prep", "D": 1025, "R": 64, "P": 91, "mode": 0, "reg": "search"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fbp", "fbp", "radon", "radon", "tv", "tv", "ragged", "grad", "prep"])
    if kind in ("fbp", "radon", "tv"):
        # grids are odd for an even detector (one bin is added) and even after sub-sampling
        N, T = _log(rng, 97, 2049), _log(rng, 60, 1500)
        top = 256 * 1200 * 2049 ** 2 // (4 if kind != "tv" else 24)
        S = _log(rng, 1, max(1, min(256, top // (T * N * N))))
        c = {"kind": kind, "N": N, "T": T, "S": S, "closed": rng.random() < 0.5}
        if kind == "tv":
            c.update(nouter=rng.choice([1, 1, 2]), ncg=rng.choice([2, 3, 4]))
        return c
    if kind == "ragged":
        return {"kind": kind, "P": rng.randint(2, 9), "Nmax": _log(rng, 129, 1449), "Tmax": _log(rng, 90, 900),
                "nouter": 1, "ncg": rng.choice([2, 3])}
    if kind == "grad":
        N, T = _log(rng, 97, 1449), _log(rng, 60, 900)
        return {"kind": kind, "N": N, "T": T, "S": max(1, min(4, 2 * 750 * 1025 ** 2 // (T * N * N)))}
    reg = rng.choice(["xcorr", "search"])
    return {"kind": kind, "D": _log(rng, 256, 2048), "R": _log(rng, 16, 256), "P": rng.randint(30, 180),
            "mode": rng.choice([0, 1]), "reg": reg}


# ---- inputs --------------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) % (1 << 31))
    return g


def _theta(T, closed):
    n = T - 1 if closed and T > 1 else T
    return (np.arange(T, dtype=np.float64) * (180.0 / n)).astype(np.float32)


def _ellipses(seed, radius, n=10):
    """Ten ellipses: centres in the disc, semi-axes 0.05-0.4 of the radius, attenuation 0.1-1.0, height of their middle."""
    r = np.random.default_rng(int(seed))
    out = []
    for _ in range(n):
        d, p = radius * math.sqrt(r.uniform()), r.uniform(0, 2 * math.pi)
        a, b = r.uniform(0.05, 0.4, 2) * radius
        out.append((d * math.cos(p), d * math.sin(p), a, b, r.uniform(0, math.pi), r.uniform(0.1, 1.0), r.uniform(0, 1)))
    return out


def _heights(S, z):
    """Squared relative axes of an ellipsoid's cut in each of S slices."""
    s = (torch.arange(S, device=DEV, dtype=torch.float32) + 0.5) / S
    return torch.clamp(1.0 - ((s - z) / 0.9) ** 2, min=0.02)


def _phantom(seed, N, S):
    m = (N + 1) // 2
    j = torch.arange(1, N + 1, device=DEV, dtype=torch.float32) - m
    Y, X = torch.meshgrid(j, j, indexing="ij")
    img = torch.zeros(S, N, N, device=DEV)
    for cx, cy, a, b, phi, v, z in _ellipses(seed, 0.35 * N):
        c, s = math.cos(phi), math.sin(phi)
        q = ((c * (X - cx) + s * (Y - cy)) / a) ** 2 + ((c * (Y - cy) - s * (X - cx)) / b) ** 2
        f = _heights(S, z)
        for k in range(S):
            img[k] += v * (q <= f[k])
    return img


def _line_integrals(seed, N, theta, S, det_offset=0.0, nbins=None):
    """[S][T][bins]: the phantom's integrals along the rays the projector samples, over N."""
    m = (N + 1) // 2
    ct = (torch.as_tensor(theta, device=DEV).double() - 90.0) * (math.pi / 180.0)
    c, s = torch.cos(ct)[:, None], torch.sin(ct)[:, None]
    off = torch.arange(1, (nbins or N) + 1, device=DEV, dtype=torch.float64)[None, :] - m - det_offset
    out = torch.zeros(S, len(theta), nbins or N, device=DEV)
    for cx, cy, a, b, phi, v, z in _ellipses(seed, 0.35 * N):
        cp, sp = math.cos(phi), math.sin(phi)
        px, py = -s * off - cx, c * off - cy
        qx, qy = (cp * px + sp * py) / a, (cp * py - sp * px) / b
        ex, ey = (cp * c + sp * s) / a, (cp * s - sp * c) / b
        A, B, C = ex * ex + ey * ey, 2 * (qx * ex + qy * ey), qx * qx + qy * qy
        base, slope, scale = (B * B - 4 * A * C).float(), (4 * A).float(), (v / (N * A)).float()
        f = _heights(S, z)
        for k in range(S):
            out[k] += torch.sqrt(torch.clamp(base + slope * f[k], min=0.0)) * scale
    return out


def _sinograms(seed, N, theta, S):
    """Log-normalised Poisson counts."""
    p = _line_integrals(seed, N, theta, S)
    g = _gen(seed)
    for k in range(S):
        p[k] = -torch.log(torch.clamp(torch.poisson(I0 * torch.exp(-p[k]), generator=g), min=1.0) / I0)
    return p


def _wpu(N):
    return max(4, N // 20)


def _ragged_problems(case):
    """Sides and angle counts of the problems of a ragged batch: the sides step down from the largest, angles vary."""
    out = []
    for k in range(case["P"]):
        f = (1.0, 0.25, 0.71, 0.5, 0.354, 0.9, 0.6, 0.18, 0.8)[k % 9]
        g = (0.4, 1.0, 0.68, 0.2, 0.85, 0.33, 0.55, 0.9, 0.25)[k % 9]
        out.append((max(33, int(case["Nmax"] * f) | 1), max(20, int(case["Tmax"] * g))))
    return out


def _counts(case, seed):
    """Raw projections of a row-by-row phantom, flat and dark frames (uint16), angles."""
    D, R, P = case["D"], case["R"], case["P"]
    Ng = D + (1 if D % 2 == 0 else 0)
    th = _theta(P, True)
    off = float(np.random.default_rng(int(seed)).uniform(-8, 8)) * min(1.0, D / 2048)
    p = _line_integrals(seed, Ng, th, R, det_offset=off, nbins=D).permute(1, 0, 2).contiguous() * (4.0 * Ng / D)
    g = _gen(seed)
    u16 = lambda x: torch.clamp(x, 0, 65535).to(torch.int32).to(torch.uint16)  # noqa: E731
    raw = u16(torch.poisson(1e4 * torch.exp(-p), generator=g) + 100.0)
    flats = u16(torch.poisson(torch.full((10, R, D), 1e4, device=DEV), generator=g) + 100.0)
    darks = u16(torch.poisson(torch.full((10, R, D), 100.0, device=DEV), generator=g))
    return th, raw, flats, darks


def _inputs(case, seed):
    k = case["kind"]
    if k == "fbp" or k == "tv":
        return {"f": _sinograms(seed, case["N"], _theta(case["T"], case["closed"]), case["S"])}
    if k == "radon":
        return {"u": _phantom(seed, case["N"], case["S"])}
    if k == "ragged":
        return {"f": [_sinograms(seed + 31 * i, N, _theta(T, False), 1)[0].cpu().numpy()
                      for i, (N, T) in enumerate(_ragged_problems(case))]}
    if k == "grad":
        g = _gen(seed)
        N, T, S = case["N"], case["T"], case["S"]
        u = _phantom(seed, N, S)
        u += 0.01 * torch.randn(u.shape, device=DEV, generator=g)
        return {"u": u, "off": 2.0 * torch.randn(S, T, device=DEV, generator=g),
                "y": _sinograms(seed + 1, N, _theta(T, False), S)}
    th, raw, flats, darks = _counts(case, seed)
    return {"th": th, "raw": raw, "flats": flats, "darks": darks}


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=dict(case))
    k = case["kind"]
    if k == "ragged":
        probs = _ragged_problems(case)
        s["h"] = RaggedBatch([n for n, _ in probs], [_theta(t, False) for _, t in probs], [_wpu(n) for n, _ in probs])
    elif k == "prep":
        s["h"] = Preprocessor()
    else:
        s["h"] = Tomography(case["N"], _theta(case["T"], case.get("closed", False)), _wpu(case["N"]))
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------

def _kmax(D):
    return max(1, min(D // 4, 512))


def run(state):
    c, h = state["case"], state["h"]
    k = c["kind"]
    if k == "fbp":
        return h.iradon(state["f"])
    if k == "radon":
        return h.radon(state["u"])
    if k == "tv":
        return h.tvopt(state["f"], 1, c["nouter"], c["ncg"], LAM, MU)
    if k == "ragged":
        return h.tvopt(state["f"], 1, c["nouter"], c["ncg"], LAM, MU)
    if k == "grad":
        return h.tv_loss_grad(state["u"], state["off"], state["y"], LAM, EPS)
    D = c["D"]
    add = 1 if D % 2 == 0 else 0
    ob, df = h.frame_average(state["flats"]), h.frame_average(state["darks"])
    proj = h.normalize(state["raw"], ob, df, c["mode"])
    p0, p180 = h.pick_angle(state["th"], proj, 0.0), h.pick_angle(state["th"], proj, 180.0)
    if c["reg"] == "xcorr":
        kb, ks, corr = h.xcorr_register(p0, p180, _kmax(D))
        return {"lag": kb, "lag_sub": ks, "corr": corr, "proj": proj,
                "sino": h.proj_to_sino(proj, 0.0, (add - ks) / (2.0 * D))}
    th, sh, ne = h.register(p0, p180)
    return {"theta": th, "shift": sh, "evals": ne, "proj": proj, "sino": h.proj_to_sino(proj, th, sh)}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _op(N, T, S):
    """Flops of one projection (four taps a sample) and of one filtered backprojection (two taps an update)."""
    return 8.0 * T * N * N * S, 4.0 * T * N * N * S


def work(case):
    k = case["kind"]
    if k == "prep":
        D, R, P = case["D"], case["R"], case["P"]
        n, nx = P * R * D, D + (1 if D % 2 == 0 else 0)
        nk = 2 * _kmax(D) + 1
        # selecting a median of 27 takes some 100 comparisons, a resampled value 11 operations, a normalised one 3
        flops = n * (3.0 + 100.0) + P * R * nx * 11.0 + (2.0 * R * D * nk if case["reg"] == "xcorr" else 0.0)
        return {"bytes": 2.0 * n + 2.0 * 20 * R * D + 4.0 * n + 4.0 * P * R * nx, "flops": flops}
    if k == "ragged":
        b = f = 0.0
        for N, T in _ragged_problems(case):
            r, i = _op(N, T, 1)
            b += 4.0 * (T * N + 2 * N * N)
            f += (1 + case["nouter"] * case["ncg"]) * (r + i)
        return {"bytes": b, "flops": f}
    N, T, S = case["N"], case["T"], case["S"]
    r, i = _op(N, T, S)
    if k == "fbp":
        return {"bytes": 4.0 * S * (T * N + N * N), "flops": i}
    if k == "radon":
        return {"bytes": 4.0 * S * (T * N + N * N), "flops": r}
    if k == "tv":
        return {"bytes": 4.0 * S * (T * N + 2 * N * N), "flops": (1 + case["nouter"] * case["ncg"]) * (r + i)}
    # the projection, its transpose and its derivative with respect to the offsets
    return {"bytes": 4.0 * S * (T * N + 2 * N * N + 2 * T), "flops": 3.0 * r}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------

F64 = torch.float64


def _samples(N, m, c, s, dy, rows):
    """Cells, bilinear weights and validity of the samples of some rays of one angle: [rays][steps]."""
    dx = (torch.arange(1, N + 1, device=DEV, dtype=F64) - m)[None, :]
    d = dy[rows][:, None]
    xr, yr = c * dx - s * d + m, s * dx + c * d + m
    x1, y1 = torch.floor(xr), torch.floor(yr)
    ok = (torch.minimum(x1, y1) > 1) & (torch.maximum(x1, y1) < N)
    i = torch.where(ok, (y1 - 1) * N + (x1 - 1), torch.zeros_like(x1)).long()
    fx, fy = xr - x1, yr - y1
    return i, fx, fy, ok.to(F64)


def _rays(N, S):
    n = max(1, (1 << 25) // (N * S))
    return [slice(a, min(a + n, N)) for a in range(0, N, n)]


def _radon64(u, theta):
    S, N = u.shape[0], u.shape[-1]
    m = (N + 1) // 2
    p = u.reshape(S, N * N).t().contiguous()
    dy = torch.arange(1, N + 1, device=DEV, dtype=F64) - m
    out = torch.empty(S, len(theta), N, device=DEV, dtype=F64)
    for t, th in enumerate(theta):
        a = math.pi * (float(th) - 90.0) / 180.0
        c, s = math.cos(a), math.sin(a)
        for rows in _rays(N, S):
            i, fx, fy, ok = _samples(N, m, c, s, dy, rows)
            v = 0.0
            for o, w in ((0, (1 - fx) * (1 - fy)), (1, fx * (1 - fy)), (N, (1 - fx) * fy), (N + 1, fx * fy)):
                j = (i + o).clamp_(max=N * N - 1)
                v = v + torch.einsum("rn,rns->rs", w * ok, p[j])
            out[:, t, rows] = v.t()
    return out / N


def _mask64(N, T, wpu):
    a = torch.arange(1, N + 1, device=DEV, dtype=F64) - (N - 1.0) / 2.0 - 1.0
    r = torch.sqrt(a[None, :] ** 2 + a[:, None] ** 2)
    q = 1.0 - 2.0 * (r - ((N - 1.0) / 2.0 - wpu)) / wpu
    mid = torch.exp(1.0 - 1.0 / (1.0 - torch.exp(1.0 - 1.0 / (1.0 - q))))
    return torch.where(q <= 0, torch.zeros_like(q), torch.where(q >= 1, torch.ones_like(q), mid)) * (math.pi / T)


def _iradon64(f, theta, wpu):
    S, T, N = f.shape
    m, L = (N + 1) // 2, 1 << (3 * N).bit_length()
    k = torch.arange(-(N - 1), N, device=DEV, dtype=F64)
    taps = -(2.0 * N) / (math.pi ** 2 * (4.0 * k * k - 1.0))
    H = torch.fft.rfft(taps, n=L)
    q = torch.empty_like(f)
    for z in range(S):
        q[z] = torch.fft.irfft(torch.fft.rfft(f[z], n=L) * H, n=L)[:, N - 1:2 * N - 1]
    q = q.permute(1, 2, 0).contiguous()
    d = torch.arange(1, N + 1, device=DEV, dtype=F64) - m
    img = torch.zeros(N, N, S, device=DEV, dtype=F64)
    rows = max(1, (1 << 26) // (N * S))
    for t, th in enumerate(theta):
        a = math.pi * (90.0 - float(th)) / 180.0
        c, s = math.cos(a), math.sin(a)
        for y in range(0, N, rows):
            yr = s * d[None, :] + c * d[y:y + rows, None] + m
            y1 = torch.floor(yr)
            ok = (y1 > 1) & (y1 < N)
            i = torch.where(ok, y1 - 1, torch.zeros_like(y1)).long()
            w = (yr - y1)[..., None]
            img[y:y + rows] += (q[t][i] * (1 - w) + q[t][(i + 1).clamp_(max=N - 1)] * w) * ok[..., None]
    return (img * _mask64(N, T, wpu)[..., None]).permute(2, 0, 1)


def _tv64(f, theta, wpu, nouter, ncg):
    lap = lambda u: 4 * u - u.roll(1, -1) - u.roll(-1, -1) - u.roll(1, -2) - u.roll(-1, -2)  # noqa: E731
    dot = lambda a, b: (a * b).sum((-1, -2), keepdim=True)                                    # noqa: E731
    ratio = lambda a, b: torch.where(b == 0, torch.zeros_like(b), a / torch.where(b == 0, torch.ones_like(b), b))  # noqa: E731
    shrink = lambda t: torch.sign(t) * torch.clamp(t.abs() - 1.0 / LAM, min=0.0)              # noqa: E731
    A = lambda u: _iradon64(_radon64(u, theta), theta, wpu)                                   # noqa: E731
    fbp = _iradon64(f, theta, wpu)
    u, fk = fbp.clone(), f.clone()
    dx = dy = bx = by = torch.zeros_like(u)
    ru = _radon64(u, theta)
    for _ in range(nouter):
        ex, ey = dx - bx, dy - by
        r = MU * _iradon64(fk - ru, theta, wpu) + LAM * (ex.roll(-1, -1) - ex + ey.roll(-1, -2) - ey) - LAM * lap(u)
        p, rs = r.clone(), dot(r, r)
        for _ in range(ncg):
            q = MU * A(p) + LAM * lap(p)
            al = ratio(rs, dot(p, q))
            u, r = u + al * p, r - al * q
            new = dot(r, r)
            p, rs = r + ratio(new, rs) * p, new
        t = u.roll(1, -1) - u + bx
        dx = shrink(t)
        bx = t - dx
        t = u.roll(1, -2) - u + by
        dy = shrink(t)
        by = t - dy
        if nouter > 1:
            ru = _radon64(u, theta)
            fk = fk + f - ru
    return u, fbp


def _grad64(u, off, y, theta):
    S, N = u.shape[0], u.shape[-1]
    T, m = len(theta), (N + 1) // 2
    loss, gu, go = torch.zeros(S, dtype=F64), torch.zeros_like(u), torch.zeros(S, T, device=DEV, dtype=F64)
    j = torch.arange(1, N + 1, device=DEV, dtype=F64) - m
    for z in range(S):
        v, acc = u[z].reshape(-1), gu[z].view(-1)
        total = torch.zeros((), device=DEV, dtype=F64)
        for t, th in enumerate(theta):
            a = math.pi * (float(th) - 90.0) / 180.0
            c, s = math.cos(a), math.sin(a)
            i, fx, fy, ok = _samples(N, m, c, s, j + off[z, t], slice(0, N))
            at = [(i + o).clamp_(max=N * N - 1) for o in (0, 1, N, N + 1)]
            w = [(1 - fx) * (1 - fy) * ok, fx * (1 - fy) * ok, (1 - fx) * fy * ok, fx * fy * ok]
            p = [v[k] for k in at]
            r = sum((a_ * b_) for a_, b_ in zip(w, p)).sum(1) / N - y[z, t]
            gx = ((p[1] - p[0]) * (1 - fy) + (p[3] - p[2]) * fy) * ok
            gy = ((p[2] - p[0]) * (1 - fx) + (p[3] - p[1]) * fx) * ok
            go[z, t] = (r * (gy * c - gx * s).sum(1) / N).sum()
            total += 0.5 * (r * r).sum()
            for k, b in zip(at, w):
                acc.index_add_(0, k.reshape(-1), (b * (r / N)[:, None]).reshape(-1))
        g = u[z]
        for dim in (-1, -2):
            d = g.roll(1, dim) - g
            n = torch.sqrt(d * d + EPS * EPS)
            total += LAM * n.sum()
            q = LAM * d / n
            gu[z] += q.roll(-1, dim) - q
        loss[z] = total.cpu()
    return loss.numpy(), gu, go


def _prep64(case, seed):
    th, raw, flats, darks = _counts(case, seed)
    wide = lambda x: x.to(torch.int32).to(F64)  # noqa: E731
    ob, df = wide(flats).mean(0), wide(darks).mean(0)
    D, R, P = case["D"], case["R"], case["P"]
    if case["mode"] == 0:
        proj = -torch.log(wide(raw) / torch.clamp(ob, min=1.0))
    else:
        proj = -torch.log(torch.clamp(wide(raw) - df, min=1e-16) / torch.clamp(ob - df, min=1.0))
    if case["reg"] != "xcorr":
        return {"theta": None, "shift": None, "evals": None, "proj": proj, "sino": None}
    # the axis: p0 against the mirrored p180, the peak refined by a parabola
    kmax, add = _kmax(D), 1 if D % 2 == 0 else 0
    p0, m180 = proj[0], proj[P - 1].flip(-1)
    corr = [float((p0[:, max(0, k):D + min(0, k)] * m180[:, max(0, -k):D - max(0, k)]).sum()) for k in range(-kmax, kmax + 1)]
    b = int(np.argmax(corr))
    frac = 0.0
    if 0 < b < 2 * kmax and corr[b - 1] - 2 * corr[b] + corr[b + 1] < 0:
        frac = 0.5 * (corr[b - 1] - corr[b + 1]) / (corr[b - 1] - 2 * corr[b] + corr[b + 1])
    shift = float(np.float32((add - (b - kmax + frac)) / (2.0 * D)))
    sino = torch.empty(R, P, D + add, device=DEV, dtype=F64)
    x = torch.arange(1, D + add + 1, device=DEV, dtype=F64) - D * shift   # no rotation: rows stay rows
    x = torch.clamp(x, 1.0, float(D))
    x1 = torch.floor(x).long()
    x2 = torch.clamp(x1 + 1, max=D)
    for k in range(P):
        three = torch.stack([proj[max(k - 1, 0)], proj[k], proj[min(k + 1, P - 1)]])
        e = torch.nn.functional.pad(three[None], (1, 1, 1, 1), mode="replicate")[0]
        n = torch.stack([e[z, a:a + R, c:c + D] for z in range(3) for a in range(3) for c in range(3)])
        med = torch.sort(n, dim=0).values[13]
        # the vertical weights are 1 and 0 except in the last row, where both taps are the row itself and weigh nothing
        v = med[:, x1 - 1] * (x2 - x) + med[:, x2 - 1] * (x - x1)
        v[R - 1] = 0.0
        sino[:, k] = v
    return {"lag": None, "lag_sub": None, "corr": None, "proj": proj, "sino": sino}


def exact(case, seed):
    k = case["kind"]
    if k == "prep":
        return _prep64(case, seed)
    x = _inputs(case, seed) if k in ("ragged", "grad") or _cost64(case) < 8e11 else None
    if x is None:
        return None
    if k == "ragged":
        tv, fbp = [], []
        for f, (N, T) in zip(x["f"], _ragged_problems(case)):
            a, b = _tv64(torch.from_numpy(f).to(DEV).to(F64)[None], _theta(T, False), _wpu(N), case["nouter"], case["ncg"])
            tv.append(a[0])
            fbp.append(b[0])
        return tv, fbp
    th = _theta(case["T"], case.get("closed", False))
    if k == "grad":
        return _grad64(x["u"].to(F64), x["off"].to(F64), x["y"].to(F64), th)
    if k == "fbp":
        return _iradon64(x["f"].to(F64), th, _wpu(case["N"]))
    if k == "radon":
        return _radon64(x["u"].to(F64), th)
    return _tv64(x["f"].to(F64), th, _wpu(case["N"]), case["nouter"], case["ncg"])


def _cost64(case):
    """Taps to gather in double precision."""
    one = float(case["N"]) ** 2 * case["T"] * (case["S"] + 8)
    if case["kind"] == "tv":
        return one * 6 * (2 + case["nouter"] * (case["ncg"] + 1))
    return one * (4 if case["kind"] == "radon" else 2)
