"""The tiles and halos of the tridiagonal column pass (unw_col_tri.cu), column by column.

The operator on white noise is dominated by its lowest modes, which hide what the fast columns (l / W >=
0.0892) contribute.  Here the input holds columns above the wide range only, and the result is compared per
column of its row DCT, with a bar that a halved halo does not meet (checked on the CPU, with the halo
planted in a float64 restatement of the tiles).  The heights lie one below, at and one above the
edges of the tiles: 128 and 192 rows for segments of 16 rows, 384 and 448 for segments of 32, which a grid
takes from 296 CTAs on; the segment length that ran is read from the kernel's name.
"""
import ctypes as C
import re

import numpy as np
import pytest
import scipy.fft as sfft
from scipy.signal import lfilter

# Two row transforms in float32, each up to two FFTs of 14 levels: 56 roundings of u = 2^-24 that add like noise,
# 4.5e-7 of a value's size, and the largest of a million such errors is 5 times that: 2.3e-6 of the rms,
# of which the largest value is at least twice; twiddle and chirp tables add about as much again.
BAR = 5e-6


def fast_columns(W):
    """The first fast columns with the long halo and with the short one: wide columns (l / W < 0.0892) come in
    groups of 32, then long-halo strips of 64 as far as l / W = 0.1821."""
    a = 32 * -(-W * 892 // 320000)
    b = a + 64 * max(0, -(-(-(-W * 1821 // 10000) - a) // 64))
    return [slice(c, min(c + 64, W)) for c in (a, b)]


def band_input(H, W, cols, seed):
    X = np.zeros((H, W))
    X[:, cols] = np.random.default_rng(seed).standard_normal((H, cols.stop - cols.start))
    return sfft.idct(X, type=2, axis=1).astype(np.float32)


def columns64(r, cols):
    """Columns of the row DCT of z in float64: column l solves (T_H + 4 sin^2(pi l / 2W)) z = x."""
    H, W = r.shape
    x = sfft.dct(r.astype(np.float64), type=2, axis=1)[:, cols]
    lam = (4 * np.sin(np.pi * np.arange(H) / (2 * H)) ** 2)[:, None] + 4 * np.sin(
        np.pi * np.arange(cols.start, cols.stop) / (2 * W)) ** 2
    return sfft.idct(sfft.dct(x, type=2, axis=0) / lam, type=2, axis=0)


def tiled(x, rho, halo, rows):
    """The recurrences of one column over tiles of `rows` rows that see `halo` rows on either side."""
    H = len(x)
    z = np.empty(H)
    for t0 in range(0, H, rows):
        j = np.arange(t0 - halo, min(t0 + rows, H) + halo) % (2 * H)
        w = x[np.where(j < H, j, 2 * H - 1 - j)]
        f = lfilter([1.0], [1.0, -rho], w)
        b = lfilter([1.0], [1.0, -rho], w[::-1])[::-1]
        z[t0:t0 + rows] = ((f + b - w) * rho / (1 - rho * rho))[halo:len(w) - halo]
    return z


@pytest.mark.parametrize("H,W,rows", [(193, 3001, (128, 192)), (385, 3000, (128, 192)), (1345, 6401, (384, 448))])
def test_bar_tells_a_halved_halo(H, W, rows):
    for cols, halo, n in zip(fast_columns(W), (64, 32), rows):
        r = band_input(H, W, cols, H)
        x = sfft.dct(r.astype(np.float64), type=2, axis=1)[:, cols]
        z = columns64(r, cols)
        rho = np.exp(-2 * np.arcsinh(np.sin(np.pi * np.arange(cols.start, cols.stop) / (2 * W))))
        err = {h: max(np.abs(tiled(x[:, k], rho[k], h, n) - z[:, k]).max() for k in range(len(rho))) / np.abs(z).max()
               for h in (halo, halo // 2)}
        assert err[halo] <= BAR / 50 and err[halo // 2] >= 2 * BAR


def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _kernels(torch, fn):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.key for e in prof.key_averages()]


SHAPES = [(16, h, w) for h, w in [(33, 1000), (63, 1001), (64, 1024), (65, 700), (127, 1001), (128, 1000), (129, 2048),
                                  (191, 1001), (192, 1000), (193, 1001), (385, 1000), (385, 3000), (449, 2999)]]
SHAPES += [(32, h, w) for h, w in [(383, 19208), (384, 19208), (385, 19683), (447, 19683), (448, 19208), (449, 9604),
                                   (769, 9604), (1151, 6401), (1152, 6400), (1153, 6401), (1343, 6401), (1344, 6400),
                                   (1345, 6401), (2689, 4001)]]


@pytest.mark.gpu
@pytest.mark.parametrize("L,H,W", SHAPES)
def test_fast_columns_at_the_edges_of_the_tiles(L, H, W):
    torch = _gpu()
    from core_b200 import _lib
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    ws = torch.full((lib.unw_workspace_bytes(H, W),), 0xA5, dtype=torch.uint8, device=dev)
    for q, cols in enumerate(fast_columns(W)):
        r = band_input(H, W, cols, H + W)
        t = torch.from_numpy(r).to(dev)
        z = torch.full((H, W), float("nan"), dtype=torch.float32, device=dev)
        run = lambda: _lib.check(lib.unw_apply_preconditioner(t.data_ptr(), H, W, z.data_ptr(), ws.data_ptr(), ws.numel(),
                                                              torch.cuda.current_stream(dev).cuda_stream))
        if q == 0:
            names = [n for n in _kernels(torch, run) if "k_col_tri" in n]
            assert names and all(re.search(r"k_col_tri<(\(int\))?%d\b" % L, n) for n in names), names
        else:
            run()
        got = sfft.dct(z.cpu().numpy().astype(np.float64), type=2, axis=1)[:, cols]
        ref = columns64(r, cols)
        assert np.abs(got - ref).max() <= BAR * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("L,H,W", [(16, 193, 1001), (16, 1025, 700), (32, 1153, 6401), (32, 2689, 4001)])
def test_tma_tiles_equal_plain_loads(L, H, W):
    # tiles of 16 L rows moved by TMA (one box of 256 rows, or two), or loaded by the threads: the same bits
    torch = _gpu()
    from core_b200 import _lib
    from core_b200.irls import make_params
    from core_b200.synthetic import gen_g1
    p, c, _ = gen_g1(H, W, seed=H)
    dev = torch.device("cuda", 0)
    ph, wt = (torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev) for a in (p, c))
    lib = _lib.load()
    ws = torch.empty(lib.unw_workspace_bytes(H, W), dtype=torch.uint8, device=dev)
    out = []
    for flag, tma in ((_lib.UNW_F_COL_TMA, "1|true"), (_lib.UNW_F_COL_NO_TMA, "0|false")):
        prm = make_params(max_iter=2, cg_max_iter=4)
        prm.flags |= flag
        u = torch.empty((H, W), dtype=torch.float32, device=dev)
        cc = torch.empty((H, W), dtype=torch.int16, device=dev)
        st = _lib.UnwStats()
        run = lambda: _lib.check(lib.unw_solve_f32(ph.data_ptr(), W, wt.data_ptr(), W, H, W, C.byref(prm), u.data_ptr(), W,
                                                   cc.data_ptr(), W, ws.data_ptr(), ws.numel(), C.byref(st),
                                                   torch.cuda.current_stream(dev).cuda_stream))
        names = [n for n in _kernels(torch, run) if "k_col_tri" in n]
        assert names and all(re.search(r"k_col_tri<(\(int\))?%d, (\(int\))?[012], (\(bool\))?(%s)>" % (L, tma), n)
                             for n in names), names
        assert not st.as_dict()["status"] & _lib.UNW_S_TC_TIMEOUT
        out.append((u.cpu().numpy().view(np.uint32), cc.cpu().numpy()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
