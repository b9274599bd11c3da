"""Performance cases of the planar WIDIM path, over its public entry points.

A case is a dict of plain values. `kind` names the entry point:

  pair      run_piv of one image pair (host arrays or device-resident frames)
  batch     BatchRunner.run of a prepared batch, results read back
  sequence  run_piv_sequence over a list of camera frames in host memory
  ensemble  run_piv_ensemble (sum of correlation) of device-resident pairs
  sweep     one WIDIM sweep hook by hook (DeviceSession), as a host-driven
            pass loop issues it: stage, deform, correlate with uncertainty
  adjoint   NCCLoss loss and gradient of a predictor field

Images are synthetic particle images rendered on the GPU from the seed:
Gaussian particles (sigma 0.65 px, intensity U[0.5, 1]) at uniform positions,
additive noise, clamped at zero. Sizes follow the repository's own
configurations (512^2, 768 x 1024, 1024^2, 2048^2, 4096^2) and ragged ones
between them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hammerhead.jl_b200"))
import hammerhead_b200 as hb  # noqa: E402
from hammerhead_b200 import adjoint, hooks  # noqa: E402

FIELDS = ("u", "v", "peak_ratio", "correlation_moment", "uncertainty_u", "uncertainty_v")


# --- the cases --------------------------------------------------------------
def _case(name, kind, rows, cols, schedule, **kw):
    c = dict(name=name, kind=kind, rows=rows, cols=cols, schedule=schedule, flow="shear", host=False, u16=False,
             mask=False, pairs=1, ppp=0.05, noise=0.01)
    c.update(kw)
    return c


def listed():
    return [
        # a preview of one small frame, single pass: latency and launches
        _case("pair_256", "pair", 256, 256, "plain", flow="uniform"),
        # the plain method on host arrays (512 x 512, uniform displacement)
        _case("pair_512_host", "pair", 512, 512, "plain", flow="uniform", host=True),
        # the accuracy schedule on one 1024 x 1024 vortex
        _case("pair_1024_accuracy", "pair", 1024, 1024, "64-32-16", flow="vortex"),
        # a ragged frame with a static mask, rectangular windows, the
        # exclusion finder and the nine-point fit
        _case("pair_ragged_rect", "pair", 771, 1030, "rect", mask=True),
        # the highest preset effort on one 2048 x 2048 frame (256-point FFTs)
        _case("pair_2048_high", "pair", 2048, 2048, "high", flow="vortex"),
        # enlarged search area, phase correlation: large displacements in one pass
        _case("pair_search_phase", "pair", 1000, 1237, "search", flow="uniform"),
        # a stream of mixed cameras: 24 pairs of 512 x 512, 24 of 768 x 1024, 16 of 2048 x 2048
        _case("batch_mixed", "batch", 0, 0, "mixed", pairs=64),
        # chained 12-bit frames of a large camera, 75 % overlap, device-resident
        _case("series_4096_u16", "batch", 4096, 4096, "series", flow="channel", u16=True, pairs=2, ppp=0.01, noise=0.05),
        # a recording in host memory, analysed as it is copied in
        _case("sequence_1024_u16", "sequence", 1024, 1280, "64-32", flow="channel", host=True, u16=True, pairs=8),
        # sum-of-correlation ensemble of eight sparse pairs
        _case("ensemble_1024", "ensemble", 1024, 1024, "64-32-16", flow="channel", pairs=8, ppp=0.01, noise=0.05),
        # one sweep of a host-driven pass loop on a 2048 x 2048 pair
        _case("sweep_2048", "sweep", 2048, 2048, "32"),
        # differentiation: loss and gradient over a 127 x 127 predictor
        _case("adjoint_1024", "adjoint", 1024, 1024, "16", flow="vortex"),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: frames of 128 to 2600 rows and columns,
    the schedules in use, batches, sequences, ensembles, sweeps, adjoints."""
    kind = rng.choice(["pair", "pair", "pair", "batch", "batch", "sequence", "ensemble", "sweep", "adjoint"])
    flow = rng.choice(["uniform", "shear", "vortex", "channel"])
    kw = dict(flow=flow, ppp=rng.choice([0.02, 0.035, 0.05]), noise=rng.choice([0.005, 0.01, 0.03]))
    if kind == "pair":
        sched = rng.choice(["plain", "64-32", "64-32-16", "48-24", "high", "rect", "search", "series"])
        lo = 256 if sched in ("high", "series", "search") else 128
        host = rng.random() < 0.3
        c = _case("", kind, _side(rng, lo, 2600), _side(rng, lo, 2600), sched, host=host, mask=rng.random() < 0.25, **kw)
    elif kind == "batch":
        n = rng.randint(2, 12)
        c = _case("", kind, _side(rng, 192, 1600), _side(rng, 192, 1600), rng.choice(["64-32", "64-32-16", "48-24"]),
                  u16=rng.random() < 0.4, pairs=n, **kw)
    elif kind == "sequence":
        c = _case("", kind, _side(rng, 256, 1400), _side(rng, 256, 1400), rng.choice(["64-32", "48-24"]), host=True,
                  u16=rng.random() < 0.6, pairs=rng.randint(3, 9), **kw)
    elif kind == "ensemble":
        c = _case("", kind, _side(rng, 256, 1400), _side(rng, 256, 1400), rng.choice(["64-32", "64-32-16"]),
                  pairs=rng.randint(2, 8), **kw)
    elif kind == "sweep":
        c = _case("", kind, _side(rng, 256, 2200), _side(rng, 256, 2200), rng.choice(["64", "48", "32", "24", "16"]), **kw)
    else:
        c = _case("", kind, _side(rng, 256, 1800), _side(rng, 256, 1800), rng.choice(["16", "24", "32"]), **kw)
    del c["name"]
    return c


def _passes(schedule):
    final = dict(max_iterations=3, uncertainty=True)
    accurate = dict(padding=True, apodization="gauss")
    if schedule == "plain":
        return [hb.PIVParameters()]
    if schedule == "64-32":
        return hb.effort_schedule("medium")
    if schedule == "64-32-16":
        return hb.multipass_parameters([64, 32, 16], final=final, **accurate)
    if schedule == "48-24":
        return hb.multipass_parameters([48, 24], final=final, **accurate)
    if schedule == "high":
        return hb.effort_schedule("high")
    if schedule == "series":
        return hb.multipass_parameters([128, 64, 32]) + [
            hb.PIVParameters(window_size=16, overlap=12, max_iterations=3, uncertainty=True)]
    if schedule == "rect":
        return hb.multipass_parameters([(48, 32), (24, 16)], peak_finder="exclusion", subpixel_method="gauss9",
                                       final=dict(uncertainty=True), **accurate)
    if schedule == "search":
        return [hb.PIVParameters(window_size=32, search_area_size=64, overlap=16, correlation_method="phase")]
    return [hb.PIVParameters(window_size=int(schedule), overlap=int(schedule) // 2, uncertainty=True, **accurate)]


def _shapes(case):
    """(rows, cols, schedule) of every pair."""
    if case["schedule"] != "mixed":
        return [(case["rows"], case["cols"], case["schedule"])] * case["pairs"]
    sizes = [(512, 512)] * 24 + [(768, 1024)] * 24 + [(2048, 2048)] * 16
    return [(r, c, ("64-32-16", "48-24")[i % 2]) for i, (r, c) in enumerate(sizes)]


# --- inputs -----------------------------------------------------------------
def _flow(kind, rows, cols, rng):
    """Displacement (u, v) at (x, y), pixels, as a function of torch tensors."""
    if kind == "uniform":
        a, b = rng.uniform(-4, 4, 2)
        return lambda x, y: (torch.full_like(x, a), torch.full_like(y, b))
    if kind == "shear":
        a, lam, ph = rng.uniform(1, 6), rng.uniform(128, 512), rng.uniform(0, 6.28)
        return lambda x, y: (a * torch.sin(2 * math.pi * y / lam + ph), torch.zeros_like(y))
    if kind == "channel":
        a = rng.uniform(4, 6)
        return lambda x, y: (a * (1 - ((y - (rows + 1) / 2) / (rows / 2)) ** 2), torch.zeros_like(y))
    rc, peak = min(rows, cols) * 0.08, rng.uniform(5, 8)
    gamma = peak * rc / 0.638173  # the largest (1 - exp(-s^2)) / s is 0.638173

    def vortex(x, y):
        dx, dy = x - (cols + 1) / 2, y - (rows + 1) / 2
        r2 = (dx * dx + dy * dy).clamp_min(1e-9)
        k = gamma / r2 * (1 - torch.exp(-r2 / rc ** 2))
        return -k * dy, k * dx
    return vortex


def _render(rows, cols, y, x, inten, noise, gen):
    """Column-major float32 (rows, cols) frame; intensities are accumulated as
    integers, so that the image does not depend on the order of the sums."""
    s = 0.65
    acc = torch.zeros(cols * rows, dtype=torch.int64, device="cuda")
    y0, x0 = torch.round(y), torch.round(x)
    ty = torch.stack([torch.exp(-((y0 + a - y) ** 2) / (2 * s * s)) for a in range(-2, 3)])
    tx = torch.stack([torch.exp(-((x0 + b - x) ** 2) / (2 * s * s)) for b in range(-2, 3)]) * inten
    iy, ix = y0.long() - 1, x0.long() - 1
    for a in range(5):
        for b in range(5):
            i, j = iy + a - 2, ix + b - 2
            ok = (i >= 0) & (i < rows) & (j >= 0) & (j < cols)
            val = torch.round(ty[a] * tx[b] * 2.0 ** 32).long()
            acc.index_add_(0, torch.where(ok, j * rows + i, 0), torch.where(ok, val, 0))
    img = acc.double() / 2.0 ** 32
    img = img + noise * torch.randn(cols * rows, generator=gen, device="cuda", dtype=torch.float32)
    return img.clamp_min(0.0).float().reshape(cols, rows).T


def _frames(case, rows, cols, seed, count):
    """`count` chained frames: the particles move by the flow from one to the next."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    flow = _flow(case["flow"], rows, cols, np.random.default_rng(seed))
    m = 12.0
    n = int(case["ppp"] * (rows + 2 * m) * (cols + 2 * m))
    p = torch.rand(3, n, generator=gen, device="cuda", dtype=torch.float64)
    y, x, inten = 1 - m + p[0] * (rows + 2 * m - 1), 1 - m + p[1] * (cols + 2 * m - 1), 0.5 + 0.5 * p[2]
    out = []
    for _ in range(count):
        img = _render(rows, cols, y, x, inten, case["noise"], gen)
        if case["u16"]:  # 12-bit counts
            img = torch.round(img.clamp(0, 1) * 4095).T.to(torch.int32).to(torch.uint16).T
        out.append(img)
        du, dv = flow(x, y)
        x, y = x + du, y + dv
    return out


def _mask(rows, cols):
    """A static body: a disc and a strip along one edge (column-major uint8)."""
    y, x = torch.meshgrid(torch.arange(rows, device="cuda"), torch.arange(cols, device="cuda"), indexing="ij")
    r = min(rows, cols) * 0.12
    m = ((y - 0.6 * rows) ** 2 + (x - 0.4 * cols) ** 2 < r * r) | (y < rows * 0.04)
    return m.to(torch.uint8).T.contiguous().T


def _host(t):
    return np.asfortranarray(t.T.cpu().numpy().T)


def _pairs(case, seed):
    shapes = _shapes(case)
    if case["kind"] in ("batch", "sequence") and case["flow"] == "channel" and len(set(shapes)) == 1:
        f = _frames(case, case["rows"], case["cols"], seed, len(shapes) + 1)  # a chained recording
        pairs = [(f[k], f[k + 1]) for k in range(len(shapes))]
    else:
        pairs = [tuple(_frames(case, r, c, seed * 1009 + i, 2)) for i, (r, c, _) in enumerate(shapes)]
    return [(_host(a), _host(b)) for a, b in pairs] if case["host"] else pairs


def _predictor(case, y, x, seed, noise):
    """The true field on nodes (y, x) plus N(0, noise) px: (2, gnx, gny) float32,
    the library's plane layout."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    flow = _flow(case["flow"], case["rows"], case["cols"], np.random.default_rng(seed * 1009))
    X, Y = torch.meshgrid(torch.as_tensor(x, dtype=torch.float64, device="cuda"),
                          torch.as_tensor(y, dtype=torch.float64, device="cuda"), indexing="ij")
    P = torch.stack(flow(X, Y))
    return (P + noise * torch.randn(P.shape, generator=gen, device="cuda", dtype=torch.float64)).float()


def prepare(case, seed):
    passes = [_passes(s) for _, _, s in _shapes(case)]
    ws = hb.piv_workspace()
    s = dict(kind=case["kind"], ws=ws, pairs=_pairs(case, seed), passes=passes[0], mask=None)
    rows, cols = case["rows"], case["cols"]
    if case["mask"]:
        m = _mask(rows, cols)
        s["mask"] = _host(m) if case["host"] else m
    if case["kind"] == "batch":
        s["runner"] = hb.BatchRunner(s["pairs"], passes, workspace=ws)
    if case["kind"] in ("sweep", "adjoint"):
        p = passes[0][0]
        x, y, _, jobs = hb.pass_grid((rows, cols), p)
        P = _predictor(case, y, x, seed, 0.3 if case["kind"] == "adjoint" else 0.05)
        A, B = (_host(t) for t in s["pairs"][0])
        if case["kind"] == "sweep":
            pu, pv = (_host(t.T) for t in P)
            s.update(A=A, B=B, x=x, y=y, jobs=jobs, pu=pu, pv=pv, session=hooks.DeviceSession(ws))
        else:
            w = p.window_size[0]
            s.update(loss=hb.NCCLoss(A, B, window=w, overlap=w // 2, workspace=ws), P=P.contiguous(),
                     grad=torch.empty_like(P), n=(len(y), len(x)),
                     grid=(float(y[0]), float(y[1] - y[0]), float(x[0]), float(x[1] - x[0])))
    return s


def _result(r):
    return {**{k: getattr(r, k) for k in FIELDS}, "outliers": r.outliers}


def run(state):
    kind, ws = state["kind"], state["ws"]
    if kind == "pair":
        A, B = state["pairs"][0]
        return _result(hb.run_piv(A, B, state["passes"], mask=state["mask"], workspace=ws))
    if kind == "batch":
        r = state["runner"].run()
        return {**{k: r.out[k] for k in FIELDS}, "outliers": r.outliers, "sweeps": r.sweeps}
    if kind == "sequence":
        res = hb.run_piv_sequence(state["pairs"], state["passes"], batch_size=4, workspace=ws)
        return [[r.u, r.v, r.peak_ratio, r.correlation_moment, r.outliers] for r in res]
    if kind == "ensemble":
        return _result(hb.run_piv_ensemble(state["pairs"], state["passes"], workspace=ws))
    if kind == "sweep":
        d = state["session"]
        d.stage_pair(state["A"], state["B"])
        y, x = state["y"], state["x"]
        nu, nv, _, _ = d.apply_predictor(state["pu"], state["pv"], y, x, y, x)
        out, locs, uq = d.process_windows(state["passes"][0], state["jobs"], want_locs=True, want_uq=True)
        return {"node_u": nu, "node_v": nv, "moved": out[:, :2], "ratio": out[:, 2], "moment": out[:, 3],
                "found": out[:, 4], "alternatives": out[:, 5:], "locs": locs, "uq": uq}
    gny, gnx = state["n"]
    loss = state["loss"].device_value_and_grad(state["P"], gny, gnx, state["grid"], state["grad"])
    return {"loss": loss, "grad": state["grad"]}


# --- what a pass cannot do without ------------------------------------------
def _grid_size(rows, cols, p):
    n = [0, 0]
    for d, ext in enumerate((rows, cols)):
        w, s, step = p.window_size[d], p.search_area_size[d], p.window_size[d] - p.overlap[d]
        n[d] = (ext - s) // step + 1
    return n[0] * n[1]


def _pass_flops(rows, cols, p, uq):
    """Three real 2-D FFTs and the spectrum product per window, and the
    Wieneke sums where the pass estimates uncertainty."""
    f = 2 if p.padding else 1
    m = f * p.search_area_size[0] * f * p.search_area_size[1]
    w = p.window_size[0] * p.window_size[1]
    return _grid_size(rows, cols, p) * (7.5 * m * math.log2(m) + 8 * m + (2 * 44 * 2 * w if uq else 0))


def work(case):
    """Inputs read once and outputs written once; every pass's windows, twice
    where it iterates to convergence, and the deformations between."""
    nbytes = flops = 0.0
    for r, c, sched in _shapes(case):
        passes = _passes(sched)
        nbytes += 2 * r * c * (2 if case["u16"] else 4) + 25 * _grid_size(r, c, passes[-1])
        if case["kind"] == "adjoint":
            flops += r * c * 700 + _grid_size(r, c, passes[0]) * passes[0].window_size[0] ** 2 * 16
            continue
        for k, p in enumerate(passes):
            sweeps = min(2, p.max_iterations) if case["kind"] != "ensemble" else 1
            flops += sweeps * _pass_flops(r, c, p, False)
            flops += (sweeps - (k == 0)) * 120 * r * c + (20 * r * c if k == 1 else 0)
        if passes[-1].uncertainty:
            flops += _pass_flops(r, c, passes[-1], True) - _pass_flops(r, c, passes[-1], False)
        if case["kind"] == "sweep":
            nbytes += 16 * _grid_size(r, c, passes[0]) * 12 + 700 * _grid_size(r, c, passes[0])
            flops += 140 * r * c
    return {"bytes": nbytes, "flops": flops}


# --- the same in 64 bits ----------------------------------------------------
def _spline64(img):
    """Cubic B-spline coefficients of a frame with one line of padding on every
    side: interpolation inside, zero second difference at the ends."""
    def solve(n):
        M = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        i = torch.arange(1, n - 1, device="cuda")
        M[i, i - 1] = M[i, i + 1] = 1 / 6
        M[i, i] = 4 / 6
        for e in (0, n - 1):
            k = [e, abs(e - 1), abs(e - 2)]
            M[e, k[0]], M[e, k[1]], M[e, k[2]] = 1, -2, 1
        return torch.linalg.inv(M)
    p = torch.nn.functional.pad(img, (1, 1, 1, 1))
    return solve(p.shape[0]) @ p @ solve(p.shape[1]).T


def _weights64(d):
    c = 1 - d
    return c ** 3 / 6, 2 / 3 - d * d + d ** 3 / 2, 2 / 3 - c * c + c ** 3 / 2, d ** 3 / 6


def _sample64(C, y, x):
    """Cubic B-spline sample at 1-based (y, x), zero outside the frame."""
    nr, nc = C.shape[0] - 2, C.shape[1] - 2
    inside = (y >= 1) & (y <= nr) & (x >= 1) & (x <= nc)
    iy = y.detach().floor().clamp(1, nr - 1)
    ix = x.detach().floor().clamp(1, nc - 1)
    wy, wx = _weights64(y - iy), _weights64(x - ix)
    iy, ix = iy.long(), ix.long()
    s = 0
    for a in range(4):
        for b in range(4):
            s = s + wy[a] * wx[b] * C[iy - 1 + a, ix - 1 + b]
    return torch.where(inside, s, torch.zeros((), dtype=s.dtype, device=s.device))


def _axis64(q, q0, step, n):
    t = ((q - q0) / step).clamp(0, n - 1)
    i = t.floor().clamp(max=n - 2).long()
    return i, t - i


def _bilinear64(f, y, x, grid):
    """f (2, gny, gnx) on uniform nodes at rows y and columns x, flat outside."""
    iy, dy = _axis64(y, grid[0], grid[1], f.shape[1])
    ix, dx = _axis64(x, grid[2], grid[3], f.shape[2])
    g = f[:, iy] * (1 - dy)[None, :, None] + f[:, iy + 1] * dy[None, :, None]
    return g[:, :, ix] * (1 - dx) + g[:, :, ix + 1] * dx


def _deform64(A, B, f, grid):
    rows, cols = A.shape
    y = torch.arange(1, rows + 1, dtype=torch.float64, device="cuda")
    x = torch.arange(1, cols + 1, dtype=torch.float64, device="cuda")
    u, v = _bilinear64(f, y, x, grid) / 2
    Y, X = y[:, None], x[None, :]
    return _sample64(_spline64(A), Y - v, X - u), _sample64(_spline64(B), Y + v, X + u)


def _apod64(p):
    w = torch.ones(p.window_size, dtype=torch.float64, device="cuda")
    if p.apodization == "gauss":
        g = [torch.exp(-((torch.arange(1, n + 1, dtype=torch.float64, device="cuda") - (n + 1) / 2) ** 2)
                       / (2 * (n / 4) ** 2)) for n in p.window_size]
        w = g[0][:, None] * g[1][None, :]
    return w


def _windows64(img, p, r0, c0, size):
    """(n, size, size) windows whose top-left pixels are (r0, c0), 0-based."""
    i = torch.arange(size[0], device="cuda")
    j = torch.arange(size[1], device="cuda")
    return img[(r0[:, None] + i)[:, :, None], (c0[:, None] + j)[:, None, :]]


def _peaks64(R, count):
    """The `count` largest positive regional maxima: (values, rows, columns),
    and how many there are."""
    n, nr, nc = R.shape
    pad = torch.nn.functional.pad(R, (1, 1, 1, 1), value=-math.inf)
    top = torch.ones_like(R, dtype=torch.bool)
    for a in range(3):
        for b in range(3):
            if (a, b) != (1, 1):
                q = pad[:, a:a + nr, b:b + nc]
                top &= (q <= R) if (b < 1 or (b == 1 and a < 1)) else (q < R)
    v, k = torch.where(top & (R > 0), R, torch.zeros_like(R)).reshape(n, -1).topk(count, dim=1)
    return v, k // nc, k % nc, (v > 0).sum(1)


def _gauss3_64(R, r, c):
    """Three-point Gaussian fit per axis around (r, c); 1-based."""
    n, nr, nc = R.shape
    j = torch.arange(n, device="cuda")
    z = R[j, r, c]

    def axis(m, p, edge):
        m, p = torch.where(edge, z, m), torch.where(edge, z, p)
        ok = ~edge & (m > 0) & (p > 0) & (z > 0)
        lm, lz, lp = (torch.log(t.clamp_min(1e-300)) for t in (m, z, p))
        den = lm - 2 * lz + lp
        return torch.where(ok & (den != 0), (lm - lp) / (2 * den), torch.zeros_like(z))
    er, ec = (r == 0) | (r == nr - 1), (c == 0) | (c == nc - 1)
    dr = axis(R[j, (r - 1).clamp_min(0), c], R[j, (r + 1).clamp_max(nr - 1), c], er)
    dc = axis(R[j, r, (c - 1).clamp_min(0)], R[j, r, (c + 1).clamp_max(nc - 1)], ec)
    return r + 1 + dr, c + 1 + dc


def _correlate64(A, B, p, r0, c0):
    """Per window: displacement, peak ratio, moment, peaks found, alternatives
    (n, 2, K-1); cross or phase correlation, regional maxima, gauss3, K = 3."""
    (wr, wc), (sr, sc) = p.window_size, p.search_area_size
    f = 2 if p.padding else 1
    nr, nc = f * sr, f * sc
    ap = _apod64(p)
    wa = _windows64(A, p, r0, c0, (wr, wc))
    wa = ap * (wa - wa.mean((1, 2), keepdim=True))
    orow, ocol = (sr - wr) // 2, (sc - wc) // 2
    wb = _windows64(B, p, r0 - orow, c0 - ocol, (sr, sc))
    wb = wb - wb.mean((1, 2), keepdim=True)
    if (sr, sc) == (wr, wc):
        wb = ap * wb
    wa = torch.nn.functional.pad(wa, (ocol, nc - wc - ocol, orow, nr - wr - orow))
    S = torch.conj(torch.fft.fft2(wa)) * torch.fft.fft2(wb, s=(nr, nc))
    if p.correlation_method == "phase":
        fr, fc = (torch.fft.fftfreq(n, 1 / n, dtype=torch.float64, device="cuda") for n in (nr, nc))
        S = S / (S.abs() + 1.1920929e-7)
        S = S * torch.exp(-(fr[:, None] ** 2 + fc[None, :] ** 2) / (2 * (min(nr, nc) / 8) ** 2))
    R = torch.fft.fftshift(torch.fft.ifft2(S).real.abs(), dim=(1, 2))
    if p.padding and (sr, sc) == (wr, wc):
        o = torch.fft.fftshift(torch.fft.ifft2(torch.fft.fft2(ap, s=(nr, nc)).abs() ** 2).real)
        R = R * torch.where(o >= o.max() / 2, o.max() / o, torch.zeros_like(o))
    if (sr, sc) != (wr, wc):
        i = (torch.arange(nr, device="cuda") - nr // 2).abs() <= orow
        j = (torch.arange(nc, device="cuda") - nc // 2).abs() <= ocol
        R = R * (i[:, None] & j[None, :])
    K = 3
    v, r, c, found = _peaks64(R, K)
    nan = torch.full_like(v[:, 0], math.nan)
    pr, pc = _gauss3_64(R, r[:, 0], c[:, 0])
    ratio = torch.where(found >= 2, v[:, 0] / v[:, 1], torch.where(found == 1, math.inf, nan))
    ri, ci = pr.round().long(), pc.round().long()
    w = sx = 0
    pad = torch.nn.functional.pad(R, (1, 1, 1, 1))
    j = torch.arange(len(R), device="cuda")
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            q = pad[j, ri + a, ci + b]
            w = w + q
            sx = sx + q * ((ri + a - pr) ** 2 + (ci + b - pc) ** 2)
    alts = []
    for m in range(1, K):
        ar, ac = _gauss3_64(R, r[:, m], c[:, m])
        alts.append(torch.stack([torch.where(found > m, ac - (nc // 2 + 1), nan),
                                 torch.where(found > m, ar - (nr // 2 + 1), nan)], 1))
    none = found == 0
    return (torch.where(none, nan, pc - (nc // 2 + 1)), torch.where(none, nan, pr - (nr // 2 + 1)), ratio,
            torch.where(none, nan, torch.sqrt(sx / w)), found.double(), torch.stack(alts, 2))


def _uq64(A, B, p, r0, c0):
    """The 2 x 44 Wieneke sums per window: C0, C+, C-, S00 and the covariances
    at the 40 half-plane lags in ring order, for u (columns) and v (rows)."""
    lags = [(dr, dc) for dc in range(5) for dr in (range(1, 5) if dc == 0 else range(-4, 5))]
    lags.sort(key=lambda o: max(abs(o[0]), o[1]))
    ap = _apod64(p)
    w = []
    for img in (A, B):
        t = _windows64(img, p, r0, c0, p.window_size)
        w.append(ap * (t - t.mean((1, 2), keepdim=True)))
    out = []
    for a, b in (w, [t.transpose(1, 2) for t in w]):
        a0, a1, b0, b1 = a[:, :, :-1], a[:, :, 1:], b[:, :, :-1], b[:, :, 1:]
        out += [(a0 * b0).sum((1, 2)), (a0 * b1).sum((1, 2)), (a1 * b0).sum((1, 2))]
        d = a0 * b1 - a1 * b0
        d = (torch.cat([d[:, :, :1], d[:, :, :-1]], 2) + 2 * d + torch.cat([d[:, :, 1:], d[:, :, -1:]], 2)) / 4
        d = d - d.mean((1, 2), keepdim=True)
        out.append((d * d).sum((1, 2)))
        R, C = d.shape[1:]
        for dr, dc in lags:
            lo, hi = max(0, -dr), min(R, R - dr)
            out.append((d[:, lo:hi, :C - dc] * d[:, lo + dr:hi + dr, dc:]).sum((1, 2)))
    return torch.stack(out, 1)


def _around64(f, valid, reach):
    """The other values within `reach` of every cell, sorted, missing ones
    last as +inf; and how many there are."""
    ny, nx = f.shape
    pf = torch.nn.functional.pad(f, (reach,) * 4)
    pv = torch.nn.functional.pad(valid, (reach,) * 4)
    got, n = [], 0
    for a in range(2 * reach + 1):
        for b in range(2 * reach + 1):
            if (a, b) != (reach, reach):
                ok = pv[a:a + ny, b:b + nx]
                got.append(torch.where(ok, pf[a:a + ny, b:b + nx], math.inf))
                n = n + ok.long()
    return torch.stack(got).sort(0).values, n


def _median64(s, n):
    i = ((n - 1).clamp_min(0) // 2, (n // 2).clamp_max(len(s) - 1))
    return (s.gather(0, i[0][None])[0] + s.gather(0, i[1][None])[0]) / 2


def _spread64(s, n, m):
    d = torch.where(torch.isinf(s), math.inf, (s - m).abs()).sort(0).values
    return _median64(d, n)


def _validated64(u, v, alts, mask):
    """Normalised median test, substitution by alternative peaks and
    replacement by local medians, on the whole grid."""
    valid = ~mask
    far = torch.zeros_like(mask)
    for f in (u, v):
        s, n = _around64(f, valid, 2)
        m = _median64(s, n)
        far |= (n > 0) & valid & ((f - m).abs() / (_spread64(s, n, m) + 0.1) > 2.0)
    good = valid & ~far
    open_ = far.clone()
    new, stat = [u.clone(), v.clone()], []
    for f in (u, v):
        s, n = _around64(f, good, 2)
        m = _median64(s, n)
        stat.append((m, _spread64(s, n, m)))
    for k in range(alts.shape[-1]):
        ok = open_ & (n >= 3)
        for d in range(2):
            a = alts[..., d, k]
            ok &= torch.isfinite(a) & ((a - stat[d][0]).abs() / (stat[d][1] + 0.1) <= 2.0)
        for d in range(2):
            new[d] = torch.where(ok, alts[..., d, k], new[d])
        open_ &= ~ok
    good, left = valid & ~open_, open_.clone()
    out = [new[0].clone(), new[1].clone()]
    for reach in range(1, 7):
        got = [_around64(f, good, reach) for f in new]
        ok = left & (got[0][1] >= 3)
        for d in range(2):
            out[d] = torch.where(ok, _median64(*got[d]), out[d])
        left &= ~ok
    nan = torch.full_like(u, math.nan)
    return [torch.where(mask, nan, f) for f in out]


def _torch64(a):
    if isinstance(a, np.ndarray):
        a = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return a.double()


def exact(case, seed):
    """The pass in 64 bits, for the single passes, the sweep and the adjoint. A
    schedule of several passes has no such value: peaks, flags and sweep
    counts decided in one pass choose the inputs of the next."""
    if case["kind"] == "sweep":
        s = prepare(case, seed)
        p, jobs = s["passes"][0], torch.from_numpy(s["jobs"]).cuda().long()
        y, x = s["y"], s["x"]
        grid = (float(y[0]), float(y[1] - y[0]), float(x[0]), float(x[1] - x[0]))
        f = torch.stack([_torch64(s["pu"]), _torch64(s["pv"])])
        nodes = _bilinear64(f, torch.as_tensor(y).cuda().double(), torch.as_tensor(x).cuda().double(), grid)
        A, B = _deform64(_torch64(s["A"]), _torch64(s["B"]), f, grid)
        rows, uq = [], []
        for q in jobs.split(max(1, 2 ** 23 // (4 * p.window_size[0] ** 2))):
            r0, c0 = q[:, 2] - 1, q[:, 3] - 1
            du, dv, ratio, mom, found, alt = _correlate64(A, B, p, r0, c0)
            rows.append((torch.stack([du, dv], 1), ratio, mom, found, torch.cat([alt[:, 0], alt[:, 1]], 1)))
            uq.append(_uq64(A, B, p, r0, c0))
        out = dict(zip(("moved", "ratio", "moment", "found", "alternatives"), (torch.cat(t) for t in zip(*rows))))
        return {"node_u": nodes[0], "node_v": nodes[1], **out, "locs": None, "uq": torch.cat(uq)}
    if case["kind"] == "adjoint":
        s = prepare(case, seed)
        P = s["P"].double().requires_grad_()
        A, B = _deform64(*(_torch64(t) for t in s["pairs"][0]), P.transpose(1, 2), s["grid"])
        w = int(case["schedule"])
        a, b = (t.unfold(0, w, w // 2).unfold(1, w, w // 2).flatten(2) for t in (A, B))
        a, b = a - a.mean(2, keepdim=True), b - b.mean(2, keepdim=True)
        loss = -((a * b).sum(2) / torch.sqrt((a * a).sum(2) * (b * b).sum(2))).sum()
        loss.backward()
        return {"loss": float(loss.detach()), "grad": P.grad}
    if case["kind"] != "pair" or case["schedule"] not in ("plain", "search") or case["mask"]:
        return None
    A, B = (_torch64(t) for t in _pairs(case, seed)[0])
    p = _passes(case["schedule"])[0]
    _, _, _, jobs = hb.pass_grid(A.shape, p)
    jobs = torch.from_numpy(jobs).cuda().long()
    ny, nx = int(jobs[:, 0].max()), int(jobs[:, 1].max())
    got = [_correlate64(A, B, p, q[:, 2] - 1, q[:, 3] - 1) for q in jobs.split(4096)]
    u, v, ratio, mom, _, alts = (torch.cat(t) for t in zip(*got))
    cells = lambda t: t.reshape(nx, ny, *t.shape[1:]).transpose(0, 1)  # noqa: E731 -- jobs run down the columns
    u, v = _validated64(cells(u), cells(v), cells(alts), torch.zeros(ny, nx, dtype=torch.bool, device="cuda"))
    return {"u": u, "v": v, "peak_ratio": cells(ratio), "correlation_moment": cells(mom), "uncertainty_u": None,
            "uncertainty_v": None, "outliers": None}
