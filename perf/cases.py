"""The measured cases: what a user of this package has it do, through its public entry points.

Kinds of case (`"kind"`), each a call that an interferogram pipeline makes:

  solve      `irls_unwrap_2d` of one grid held on the GPU, with or without coherence weights
  batch      `irls_unwrap_2d_batch` of grids of different sizes (a stack of interferograms)
  chunk      `unwrap2d_chunk` of a host raster: overlapping tiles, numpy in and out
  adjoint    `irls_adjoint_batch`: the backward pass of the differentiable unwrap
  operator   `unw_apply_preconditioner` of the C interface (callers with a solver of their own)
  goldstein  the adaptive phase filter that runs before unwrapping
  link       `link_components`, which joins separately unwrapped components

`listed()` gives the fixed cases, `draw(rng)` one more of the same ranges.  Inputs are made on
the GPU from the seed.  The `fault` scenes keep reweighting for tens of iterations, so they are
run for a number of iterations (a cap with a tolerance that is not reached), as a pipeline with a
time budget does; the smooth scenes run to the default stop.
"""
import ctypes
import math

import numpy as np
import torch

import core_b200
from core_b200 import _lib

DEVICE = "cuda"


def listed():
    return [
        # one tile of a small area of interest: launches and host work are most of its time
        {"name": "solve_tile", "kind": "solve", "H": 200, "W": 180, "scene": "smooth", "weighted": True, "max_iter": 50, "tol": 1e-3},
        # a multilooked interferogram, and the grid size of the repository's own 1024 x 1024 runs
        {"name": "solve_1024", "kind": "solve", "H": 1024, "W": 1024, "scene": "smooth", "weighted": True, "max_iter": 50, "tol": 1e-3},
        # a cropped interferogram: sizes after cropping to the valid pixels are arbitrary
        {"name": "solve_ragged", "kind": "solve", "H": 1838, "W": 2750, "scene": "smooth", "weighted": True, "max_iter": 50, "tol": 1e-3},
        # no coherence at hand: uniform weights
        {"name": "solve_noweight", "kind": "solve", "H": 2048, "W": 2048, "scene": "smooth", "weighted": False, "max_iter": 50, "tol": 1e-3},
        # the repository's headline grid (fault, strong noise), under an iteration cap
        {"name": "solve_fault_4096", "kind": "solve", "H": 4096, "W": 4096, "scene": "fault", "weighted": True, "max_iter": 8, "tol": 1e-5},
        # a stack of uneven interferograms in one call
        {"name": "batch_uneven", "kind": "batch", "n": 6, "H": 1500, "W": 2400, "scene": "smooth", "max_iter": 50, "tol": 1e-3},
        # a raster on the host, unwrapped in overlapping tiles
        {"name": "chunk_host", "kind": "chunk", "H": 1500, "W": 1300, "chunk": 512, "overlap": 0.1},
        # backward pass of the differentiable unwrap for a batch of training grids, coherence held fixed
        {"name": "adjoint_768", "kind": "adjoint", "n": 2, "H": 768, "W": 768},
        # the Poisson preconditioner by itself
        {"name": "operator_odd", "kind": "operator", "H": 1500, "W": 2001},
        # filtering before unwrapping: a full scene at the default patch, a ragged one at a small patch
        {"name": "goldstein_32", "kind": "goldstein", "H": 2048, "W": 2048, "py": 32, "px": 32, "threshold": 0.5},
        {"name": "goldstein_16_odd", "kind": "goldstein", "H": 1001, "W": 1203, "py": 16, "px": 16, "threshold": 0.5},
        # joining the components of a scene broken up by water and layover
        {"name": "link_1024", "kind": "link", "H": 1024, "W": 1024, "cells": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    if u < 0.42:
        scene = "fault" if rng.random() < 0.3 else "smooth"
        H, W = _log_int(rng, 96, 3000), _log_int(rng, 96, 3000)
        if rng.random() < 0.3:
            W = 1 << max(8, min(11, W.bit_length() - 1))
        return {"kind": "solve", "H": H, "W": W, "scene": scene, "weighted": rng.random() < 0.75,
                "max_iter": 6 if scene == "fault" else 50, "tol": 1e-5 if scene == "fault" else 1e-3}
    if u < 0.52:
        return {"kind": "batch", "n": rng.randint(2, 8), "H": _log_int(rng, 200, 1800), "W": _log_int(rng, 200, 2400),
                "scene": "smooth", "max_iter": 50, "tol": 1e-3}
    if u < 0.60:
        return {"kind": "chunk", "H": _log_int(rng, 300, 1700), "W": _log_int(rng, 300, 1700),
                "chunk": rng.choice([256, 384, 512, 700]), "overlap": rng.choice([0.05, 0.1, 0.2])}
    if u < 0.70:
        return {"kind": "adjoint", "n": rng.randint(1, 4), "H": _log_int(rng, 128, 800), "W": _log_int(rng, 128, 800)}
    if u < 0.80:
        return {"kind": "operator", "H": _log_int(rng, 64, 4000), "W": _log_int(rng, 64, 4000)}
    if u < 0.92:
        p = rng.choice([8, 16, 32, 32, 64])
        return {"kind": "goldstein", "H": _log_int(rng, 150, 3000), "W": _log_int(rng, 150, 3000), "py": p,
                "px": rng.choice([p, p, max(8, p // 2)]), "threshold": rng.choice([0.5, 0.5, 0.3])}
    return {"kind": "link", "H": _log_int(rng, 400, 1300), "W": _log_int(rng, 400, 1300), "cells": rng.randint(5, 14)}


# ------------------------------------------------------------------ scenes
def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _uniform(rs, lo, hi):
    return float(lo + (hi - lo) * rs.rand())


def _holes(rs, H, W):
    """Three ellipses, about 5% of the grid, without data."""
    y = torch.arange(H, device=DEVICE, dtype=torch.float32)[:, None]
    x = torch.arange(W, device=DEVICE, dtype=torch.float32)[None, :]
    m = torch.zeros((H, W), dtype=torch.bool, device=DEVICE)
    base = 0.073 * math.sqrt(H * W)
    for _ in range(3):
        cy, cx, th = _uniform(rs, 0.1 * H, 0.9 * H), _uniform(rs, 0.1 * W, 0.9 * W), _uniform(rs, 0, math.pi)
        a, b = base * _uniform(rs, 0.7, 1.3), base * _uniform(rs, 0.7, 1.3)
        u = (x - cx) * math.cos(th) + (y - cy) * math.sin(th)
        v = (y - cy) * math.cos(th) - (x - cx) * math.sin(th)
        m |= (u / a) ** 2 + (v / b) ** 2 <= 1.0
    return m


def _truth(rs, H, W):
    """A ramp and eight Gaussian hills of up to 40 rad."""
    y = torch.arange(H, device=DEVICE, dtype=torch.float64)
    x = torch.arange(W, device=DEVICE, dtype=torch.float64)
    t = 0.02 * x[None, :].expand(H, W).clone()
    for _ in range(8):
        amp, sig = _uniform(rs, -40, 40), _uniform(rs, 50, 300)
        cy, cx = _uniform(rs, 0, H), _uniform(rs, 0, W)
        t += amp * torch.outer(torch.exp(-((y - cy) ** 2) / (2 * sig * sig)), torch.exp(-((x - cx) ** 2) / (2 * sig * sig)))
    return t


def _scene(seed, H, W, kind):
    """Wrapped phase and coherence (float32, NaN where there is no data), and the noisy truth."""
    rs, g = np.random.RandomState(seed & 0x7FFFFFFF), _gen(seed)
    t = _truth(rs, H, W)
    coh = torch.rand((H, W), generator=g, device=DEVICE, dtype=torch.float32)
    if kind == "fault":
        th, py, px = _uniform(rs, 0, math.pi), _uniform(rs, 0.3 * H, 0.7 * H), _uniform(rs, 0.3 * W, 0.7 * W)
        y = torch.arange(H, device=DEVICE, dtype=torch.float64)[:, None] - py
        x = torch.arange(W, device=DEVICE, dtype=torch.float64)[None, :] - px
        t += 3 * math.pi * ((x * math.sin(th) - y * math.cos(th)) > 0)
        coh = torch.where(coh < 0.1, torch.full_like(coh, 0.05), coh)
    else:
        coh = 0.3 + 0.7 * coh
    t += (0.6 if kind == "fault" else 0.3) * torch.randn((H, W), generator=g, device=DEVICE, dtype=torch.float32)
    wrapped = torch.atan2(torch.sin(t), torch.cos(t)).to(torch.float32)
    m = _holes(rs, H, W)
    wrapped[m] = float("nan")
    coh[m] = float("nan")
    return wrapped, coh, t


def _tiles(H, W, chunk, overlap):
    """Tiles of a raster and their halos: regular chunks extended by the overlap depth inside the
    raster, a last chunk that is shallower than the depth joined to its neighbour."""
    axes = []
    for n in (H, W):
        sizes = [min(chunk, n - a) for a in range(0, n, chunk)]
        depth = max(1, int(overlap * sizes[0]))
        if len(sizes) > 1 and sizes[-1] < depth:
            sizes[-2:] = [sizes[-2] + sizes[-1]]
        at = [sum(sizes[:i]) for i in range(len(sizes) + 1)]
        axes.append([(a, b, max(0, a - depth), min(n, b + depth)) for a, b in zip(at, at[1:])])
    return [y + x for y in axes[0] for x in axes[1]]


def _batch_sizes(c):
    """Sizes of a stack: rows and columns spread by up to 30% below the largest."""
    rs = np.random.RandomState(c["n"] * 1000003 + c["H"] * 1009 + c["W"])
    return [(max(64, int(c["H"] * (1 - 0.3 * rs.rand()))), max(64, int(c["W"] * (1 - 0.3 * rs.rand())))) for _ in range(c["n"])]


def _link_scene(seed, H, W, cells):
    """One ellipse in each cell of a lattice, every one off by its own multiple of 2 pi; labels by size."""
    rs, g = np.random.RandomState(seed & 0x7FFFFFFF), _gen(seed)
    ch, cw = H / cells, W / cells
    y = torch.arange(H, device=DEVICE, dtype=torch.float32)[:, None]
    x = torch.arange(W, device=DEVICE, dtype=torch.float32)[None, :]
    iy, ix = (y / ch).floor().clamp(max=cells - 1).long(), (x / cw).floor().clamp(max=cells - 1).long()
    par = lambda lo, hi: torch.tensor(lo + (hi - lo) * rs.rand(cells, cells), dtype=torch.float32, device=DEVICE)
    ry, rx, cy, cx = par(0.25, 0.44) * ch, par(0.25, 0.44) * cw, par(0.47, 0.53), par(0.47, 0.53)
    dy = (y - (iy + cy[iy, ix]) * ch) / ry[iy, ix]
    dx = (x - (ix + cx[iy, ix]) * cw) / rx[iy, ix]
    valid = dy * dy + dx * dx <= 1.0
    cell = torch.where(valid, iy * cells + ix + 1, torch.zeros_like(iy * cells + ix))
    size = torch.bincount(cell.reshape(-1), minlength=cells * cells + 1)
    size[0] = 1 << 30
    rank = torch.empty_like(size)
    rank[torch.argsort(size, descending=True, stable=True)] = torch.arange(size.numel(), device=DEVICE)
    shift = torch.tensor(rs.randint(-2, 3, cells * cells + 1), dtype=torch.float64, device=DEVICE)
    t = 0.03 * y.double() - 0.02 * x.double() + 2 * torch.sin(x.double() / 37) * torch.cos(y.double() / 53)
    t = t + 2 * math.pi * shift[cell] + 0.15 * torch.randn((H, W), generator=g, device=DEVICE, dtype=torch.float32)
    ph = torch.where(valid, t, torch.full_like(t, float("nan"))).to(torch.float32)
    return ph, rank[cell].to(torch.int16)


def _adjoint_inputs(c, seed):
    ph, wt, uu, gu = [], [], [], []
    for b in range(c["n"]):
        p, w, t = _scene(seed * 16 + b, c["H"], c["W"], "smooth")
        g = _gen(seed * 16 + b + 7919)
        e = torch.randn((c["H"], c["W"]), generator=g, device=DEVICE, dtype=torch.float32)
        ph.append(p)
        wt.append(w)
        uu.append((t + 0.03 * e).to(torch.float32))
        gu.append(torch.randn((c["H"], c["W"]), generator=g, device=DEVICE, dtype=torch.float32))
    return [torch.stack(v) for v in (ph, wt, uu, gu)]


# ------------------------------------------------------------------ what a user's program has in hand
def prepare(c, seed):
    k = c["kind"]
    if k == "solve":
        p, w, _ = _scene(seed, c["H"], c["W"], c["scene"])
        return {"c": c, "phase": p, "weight": w if c["weighted"] else None}
    if k == "batch":
        s = [_scene(seed * 64 + i, h, w, c["scene"])[:2] for i, (h, w) in enumerate(_batch_sizes(c))]
        return {"c": c, "phases": [p for p, _ in s], "weights": [w for _, w in s]}
    if k == "chunk":
        p, w, _ = _scene(seed, c["H"], c["W"], "smooth")
        return {"c": c, "phase": p.cpu().numpy(), "weight": w.cpu().numpy()}
    if k == "adjoint":
        return {"c": c, "in": _adjoint_inputs(c, seed)}
    if k == "operator":
        r = torch.randn((c["H"], c["W"]), generator=_gen(seed), device=DEVICE, dtype=torch.float32)
        n = _lib.load().unw_workspace_bytes(c["H"], c["W"])
        return {"c": c, "r": r, "z": torch.empty_like(r), "ws": torch.empty(n, dtype=torch.uint8, device=DEVICE)}
    if k == "goldstein":
        p, w, _ = _scene(seed, c["H"], c["W"], "smooth")
        return {"c": c, "z": torch.polar(torch.ones_like(p), p), "corr": w}
    p, lab = _link_scene(seed, c["H"], c["W"], c["cells"])
    return {"c": c, "phase": p, "lab": lab}


def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "solve":
        u, cc = core_b200.irls_unwrap_2d(s["phase"], s["weight"], max_iter=c["max_iter"], tol=c["tol"])
        return u, cc.view(torch.int16)
    if k == "batch":
        return [(u, cc.view(torch.int16)) for u, cc in
                core_b200.irls_unwrap_2d_batch(s["phases"], s["weights"], max_iter=c["max_iter"], tol=c["tol"])]
    if k == "chunk":
        return core_b200.unwrap2d_chunk(s["phase"], s["weight"], chunks=(c["chunk"], c["chunk"]), overlap=c["overlap"])
    if k == "adjoint":
        return core_b200.irls_adjoint_batch(*s["in"], need_weight=False)[0]
    if k == "operator":
        rc = _lib.load().unw_apply_preconditioner(
            ctypes.c_void_p(s["r"].data_ptr()), c["H"], c["W"], ctypes.c_void_p(s["z"].data_ptr()),
            ctypes.c_void_p(s["ws"].data_ptr()), s["ws"].numel(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.check(rc, "unw_apply_preconditioner")
        return s["z"]
    if k == "goldstein":
        return core_b200.goldstein(s["z"], s["corr"], c["py"], c["px"], c["threshold"])
    return core_b200.link_components(s["phase"], s["lab"])


def work(c):
    """Inputs once and outputs once; the operations of the method's transforms and stencils."""
    k = c["kind"]
    n = c["H"] * c["W"]
    lg = math.log2(max(2, n))
    pcg = 2 * 2.5 * lg + 40          # two 2-D DCTs and the vector work of one PCG iteration, per pixel
    if k in ("solve", "batch"):
        if k == "batch":
            n = sum(h * w for h, w in _batch_sizes(c))
        it = c["max_iter"] if c["max_iter"] < 50 else 3
        return {"bytes": (10 + (4 if c.get("weighted", True) else 0)) * n, "flops": it * 20 * pcg * n}
    if k == "chunk":
        m = n * (1 + 2 * c["overlap"]) ** 2
        return {"bytes": 12 * n, "flops": 3 * 10 * pcg * m}
    if k == "adjoint":
        return {"bytes": 20 * n * c["n"], "flops": 70 * pcg * n * c["n"]}
    if k == "operator":
        return {"bytes": 8 * n, "flops": 2 * 2.5 * lg * n}
    if k == "goldstein":
        return {"bytes": 20 * n, "flops": 4 * (2 * 5 * math.log2(c["py"] * c["px"]) + 20) * n}
    return {"bytes": 10 * n, "flops": 10 * n}


# ------------------------------------------------------------------ the same in 64 bits
def _dct(x, dim):
    x = x.movedim(dim, -1)
    n = x.shape[-1]
    v = torch.cat([x[..., ::2], x[..., 1::2].flip(-1)], -1)
    k = torch.arange(n, device=x.device, dtype=torch.float64)
    w = torch.polar(torch.ones_like(k), -math.pi * k / (2 * n))
    return (2 * torch.real(torch.fft.fft(v) * w)).movedim(-1, dim)


def _idct(y, dim):
    y = y.movedim(dim, -1)
    n = y.shape[-1]
    k = torch.arange(n, device=y.device, dtype=torch.float64)
    w = torch.polar(torch.ones_like(k), math.pi * k / (2 * n))
    m = torch.cat([torch.zeros_like(y[..., :1]), y[..., 1:].flip(-1)], -1)
    v = torch.real(torch.fft.ifft(torch.complex(y, -m) * w)) / 2
    x = torch.empty_like(v)
    h = (n + 1) // 2
    x[..., ::2] = v[..., :h]
    x[..., 1::2] = v[..., h:].flip(-1)
    return x.movedim(-1, dim)


def _precond(H, W):
    i = torch.arange(H, device=DEVICE, dtype=torch.float64)
    j = torch.arange(W, device=DEVICE, dtype=torch.float64)
    lam = (4 * torch.sin(math.pi * i / (2 * H)) ** 2)[:, None] + (4 * torch.sin(math.pi * j / (2 * W)) ** 2)[None, :]
    lam[0, 0] = 1.0

    def apply(r):
        t = _dct(_dct(r, 1), 0) / lam
        t[0, 0] = 0.0
        return _idct(_idct(t, 0), 1)

    return apply


def _grad(x):
    dx, dy = torch.zeros_like(x), torch.zeros_like(x)
    dx[:, :-1] = x[:, 1:] - x[:, :-1]
    dy[:-1] = x[1:] - x[:-1]
    return dx, dy


def _ndiv(fx, fy):
    """-div of edge values: what the transposed forward differences give."""
    r = -fx - fy
    r[:, 1:] += fx[:, :-1]
    r[1:] += fy[:-1]
    return r


def _edges(phase, weight):
    valid = ~torch.isnan(phase)
    ph = torch.where(valid, phase, torch.zeros_like(phase)).double()
    if weight is None:
        w = valid.double()
    else:
        w = torch.where(torch.isnan(weight) | ~valid, torch.zeros_like(weight), weight).double().clamp(0.01, 1.0)
        w = w.to(torch.float32).double()
    gx, gy = (torch.atan2(torch.sin(d), torch.cos(d)) for d in _grad(ph))
    wx, wy = torch.zeros_like(w), torch.zeros_like(w)
    wx[:, :-1] = (w[:, :-1] + w[:, 1:]) / 2 * (valid[:, :-1] & valid[:, 1:])
    wy[:-1] = (w[:-1] + w[1:]) / 2 * (valid[:-1] & valid[1:])
    return valid, ph, gx, gy, wx, wy


def _labels(valid):
    """4-connected components: the smallest pixel index of each, by neighbours and pointer jumps."""
    H, W = valid.shape
    n = H * W
    lab = torch.arange(n, device=valid.device).reshape(H, W)
    lab = torch.where(valid, lab, torch.full_like(lab, n))
    ext = torch.full((n + 1,), n, device=valid.device)
    for _ in range(4 * (H + W)):
        new = lab.clone()
        for a, b in ((slice(1, None), slice(None, -1)), (slice(None, -1), slice(1, None))):
            new[a] = torch.minimum(new[a], lab[b])
            new[:, a] = torch.minimum(new[:, a], lab[:, b])
        new = torch.where(valid, new, torch.full_like(new, n))
        root = ext.clone().scatter_reduce_(0, lab.reshape(-1), new.reshape(-1), "amin")
        root[n] = n
        for _ in range(3):
            root = root[root]
        new = root[torch.minimum(new, root[lab])]
        if torch.equal(new, lab):
            break
        lab = new
    return lab


def _solve64(phase, weight, max_iter, tol=1e-3, cg_max_iter=20, cg_tol=1e-4, eps=1e-2):
    """DCT-preconditioned IRLS of a grid in float64, with the median and circular-mean alignment."""
    bad = torch.isnan(phase)
    rows, cols = torch.nonzero(~bad.all(1)).reshape(-1), torch.nonzero(~bad.all(0)).reshape(-1)
    full = torch.full(phase.shape, float("nan"), dtype=torch.float64, device=phase.device)
    if rows.numel() == 0:
        return full
    r0, r1, c0, c1 = int(rows[0]), int(rows[-1]) + 1, int(cols[0]), int(cols[-1]) + 1
    phase = phase[r0:r1, c0:c1]
    weight = None if weight is None else weight[r0:r1, c0:c1]
    valid, ph, gx, gy, wx, wy = _edges(phase, weight)
    pre = _precond(*phase.shape)
    mean = lambda x: (x * valid).sum() / valid.sum()
    u = pre(_ndiv(wx * gx, wy * gy))
    u = u - mean(u)
    for _ in range(max_iter):
        prev = u
        u = u - mean(u)
        rx, ry = _grad(u)
        rx, ry = rx - gx, ry - gy
        ax = (wx / torch.sqrt(rx * rx + eps * eps)).clamp(1e-6, 1e6)
        ay = (wy / torch.sqrt(ry * ry + eps * eps)).clamp(1e-6, 1e6)

        def lap(x):
            dx, dy = _grad(x)
            return _ndiv(dx * ax, dy * ay)

        r = _ndiv(ax * gx, ay * gy) - lap(u)
        z = pre(r)
        p = z
        rz = (r * z).sum()
        for _ in range(cg_max_iter):
            q = lap(p)
            pq = (p * q).sum()
            if abs(float(pq)) < 1e-15:
                break
            alpha = (rz / pq).clamp(-1e6, 1e6)
            u = u + alpha * p
            r = r - alpha * q
            if float(torch.sqrt((r * r).sum())) < cg_tol:
                break
            z = pre(r)
            new = (r * z).sum()
            if abs(float(rz)) < 1e-15:
                break
            p = (new / rz).clamp(-1e6, 1e6) * p + z
            rz = new
        if float(torch.sqrt(((prev - u) ** 2).sum()) / (torch.sqrt((u * u).sum()) + 1e-10)) < tol:
            break
    k = torch.round((u - ph) / (2 * math.pi))[valid].sort().values
    u = u - 2 * math.pi * (k[(k.numel() - 1) // 2] + k[k.numel() // 2]) / 2
    lab = torch.unique(_labels(valid), return_inverse=True)[1].reshape(-1)
    v = valid.reshape(-1)
    tot = lambda x: torch.zeros(int(lab.max()) + 1, dtype=torch.float64, device=x.device).index_add_(
        0, lab[v], x.reshape(-1)[v])
    d = torch.atan2(tot(torch.sin(ph)), tot(torch.cos(ph))) - torch.atan2(tot(torch.sin(u)), tot(torch.cos(u)))
    u = u + torch.atan2(torch.sin(d), torch.cos(d))[lab].reshape(u.shape)
    full[r0:r1, c0:c1] = torch.where(valid, u, torch.full_like(u, float("nan")))
    return full


def _adjoint64(phase, weight, u, gu, eps=1e-2):
    """d sum(gu * out) / d phase through the solve with the IRLS scale held at u, in float64."""
    valid, ph, gx, gy, wx, wy = _edges(phase, weight)
    uf = torch.where(valid, u, torch.zeros_like(u)).double()
    dx, dy = _grad(uf)
    sx, sy = 1 / torch.sqrt((dx - gx) ** 2 + eps * eps), 1 / torch.sqrt((dy - gy) ** 2 + eps * eps)
    ax, ay = (wx * sx).clamp(1e-6, 1e6), (wy * sy).clamp(1e-6, 1e6)
    pre = _precond(*phase.shape)

    def solve(b):
        x, r = torch.zeros_like(b), b.clone()
        stop = 1e-13 * float(torch.sqrt((b * b).sum()))
        z = pre(r)
        p, rz = z, (r * z).sum()
        for _ in range(400):
            d, e = _grad(p)
            q = _ndiv(d * ax, e * ay)
            a = rz / (p * q).sum()
            x, r = x + a * p, r - a * q
            if float(torch.sqrt((r * r).sum())) < stop:
                break
            z = pre(r)
            new = (r * z).sum()
            p, rz = z + new / rz * p, new
        return x

    us = solve(_ndiv(ax * gx, ay * gy))
    lab = torch.unique(_labels(valid), return_inverse=True)[1].reshape(-1)
    v = valid.reshape(-1)
    tot = lambda x: torch.zeros(int(lab.max()) + 1, dtype=torch.float64, device=x.device).index_add_(
        0, lab[v], x.reshape(-1)[v])[lab].reshape(valid.shape)
    zero = torch.zeros_like(us)
    G = torch.where(valid, gu.double(), zero)
    S = tot(G)

    def dmean(x):
        s, c = tot(torch.sin(x)), tot(torch.cos(x))
        return (c * torch.cos(x) + s * torch.sin(x)) / (s * s + c * c)

    # through the solve: A A^+ G' = G', which sums to zero over every component
    Gp = torch.where(valid, G - S * dmean(us), zero)
    return torch.where(valid, Gp + S * dmean(ph), zero)


def _goldstein64(z, corr, py, px, threshold):
    H, W = z.shape
    sy, sx = py // 2, px // 2
    bad = torch.isnan(z.real) | torch.isnan(z.imag)
    up = lambda n, p, s: n + (p - s) + (-(n - s)) % s
    Hp, Wp = up(H, py, sy), up(W, px, sx)
    pad = lambda x: torch.nn.functional.pad(x, (0, Wp - W, 0, Hp - H))
    zero = torch.zeros_like(z)
    zz = pad(torch.where(bad, zero, z).to(torch.complex128))
    cc = pad(torch.where(torch.isnan(corr), torch.zeros_like(corr), corr).double())
    vv = pad((~bad).double())
    tent = lambda p: 1 - (torch.arange(p // 2, dtype=torch.float64, device=z.device) - (p / 2 - 1)).abs() / (p / 2 - 1)
    ty, tx = tent(py), tent(px)
    wgt = torch.outer(torch.cat([ty, ty.flip(0)]), torch.cat([tx, tx.flip(0)])).float().double()
    out, cnt = torch.zeros_like(zz), torch.zeros((Hp, Wp), dtype=torch.float64, device=z.device)
    need = int(py * px * threshold)
    for a in range(2):
        for b in range(2):
            h, w = (Hp - a * sy) // py, (Wp - b * sx) // px
            if h < 1 or w < 1:
                continue
            at = (slice(a * sy, a * sy + h * py), slice(b * sx, b * sx + w * px))
            cut = lambda x: x[at].reshape(h, py, w, px).transpose(1, 2)
            ok = cut(vv).sum((2, 3)) >= need
            alpha = 1 - (cut(cc) * wgt).sum((2, 3)) / wgt.sum()
            F = torch.fft.fft2(cut(zz))
            F = F * F.abs().clamp(min=1e-10) ** alpha[:, :, None, None]
            f = torch.fft.ifft2(F) * wgt * ok[:, :, None, None]
            out[at] += f.transpose(1, 2).reshape(h * py, w * px)
            cnt[at] += ok[:, :, None, None].double().expand(h, w, py, px).transpose(1, 2).reshape(h * py, w * px)
    r = (out / cnt.clamp(min=1))[:H, :W]
    nan = torch.complex(torch.full_like(r.real, float("nan")), torch.full_like(r.real, float("nan")))
    return torch.where(bad | (cnt[:H, :W] < 1e-6), nan, r)


def exact(c, seed):
    s = prepare(c, seed)
    k = c["kind"]
    if k == "solve":
        return _solve64(s["phase"], s["weight"], c["max_iter"], c["tol"]), None
    if k == "batch":
        return [(_solve64(p, w, c["max_iter"], c["tol"]), None) for p, w in zip(s["phases"], s["weights"])]
    if k == "chunk":
        p, w = (torch.from_numpy(s[n]).to(DEVICE) for n in ("phase", "weight"))
        out = torch.full(p.shape, float("nan"), dtype=torch.float64, device=DEVICE)
        for y0, y1, a0, a1, x0, x1, b0, b1 in _tiles(c["H"], c["W"], c["chunk"], c["overlap"]):
            u = _solve64(p[a0:a1, b0:b1], w[a0:a1, b0:b1], 50, 1e-2, 10, 1e-3)
            out[y0:y1, x0:x1] = u[y0 - a0:y1 - a0, x0 - b0:x1 - b0]
        return out.cpu().numpy()
    if k == "adjoint":
        return torch.stack([_adjoint64(*v) for v in zip(*s["in"])])
    if k == "operator":
        return _precond(c["H"], c["W"])(s["r"].double())
    if k == "goldstein":
        return _goldstein64(s["z"], s["corr"], c["py"], c["px"], c["threshold"])
    return None
