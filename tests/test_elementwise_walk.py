"""Widths and heights at the borders of the 256-column row pieces and eight-piece CTAs that the setup and
the IRLS elementwise kernels walk: the solve against the oracle at each, with the bars of the parity
tests (same NaN positions and cycle map, 1e-3 rad RMS after removal of the mean)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import core_b200  # noqa: E402
from core_b200.synthetic import gen_g1  # noqa: E402
from oracle.irls_oracle import cycle_map, irls_unwrap_2d as oracle  # noqa: E402


@pytest.mark.parametrize("H,W", [(8, 255), (9, 256), (7, 257), (33, 131), (64, 513), (257, 3)])
def test_solve_at_piece_borders(H, W):
    p, c, _ = gen_g1(H, W, seed=H + W)
    u, cc = core_b200.irls_unwrap_2d(p, c)
    uo, cco = oracle(p, c)
    v = np.isfinite(p)
    assert (np.isnan(u) == np.isnan(uo)).all()
    assert (cycle_map(u, p) == cycle_map(uo, p))[v].mean() >= 0.9999
    e = (u - uo)[v].astype(np.float64)
    assert np.sqrt(np.mean((e - e.mean()) ** 2)) <= 1e-3
    assert (cc == cco).all()


# Wrapped differences of any size stay in [-pi, pi] and are those of the exact reduction: |d| below the line
# at 1e8 (float64 reduction, rounded once: one ulp of pi), at it, and beyond, up to the largest
# float32 (float32 functions: 2 ulp of sine and cosine and 3 of the arc tangent are 1.0e-6 at pi).
# Infinite differences give NaN.
@pytest.mark.parametrize("lo,hi,tol", [(0.0, 10.0, 2.4e-7), (10.0, 1e5, 2.4e-7), (9e7, 1e8, 2.4e-7), (1e8, 1.1e8, 1.2e-6),
                                       (1e12, 1e13, 1.2e-6), (1e15, 1e17, 1.2e-6), (1e25, 3e38, 1.2e-6)])
def test_wrapped_differences_of_any_size(lo, hi, tol):
    import ctypes
    import math

    from core_b200 import _lib
    rng = np.random.default_rng(int(math.log10(hi) * 7))
    H, W = 40, 600
    p = np.zeros((H, W), np.float32)      # every other column zero: the differences are the values themselves
    p[:, 1::2] = (rng.uniform(lo, hi, (H, W // 2)) * rng.choice([-1, 1], (H, W // 2))).astype(np.float32)
    p[3, 1::2] = np.clip(np.round(p[3, 1::2].astype(np.float64) / np.pi) * np.pi, -3.4e38, 3.4e38)   # next to multiples of pi
    p[5, 7] = np.inf
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    t = torch.from_numpy(p).to(dev)
    gx, gy, wx, wy = (torch.empty((H, W), dtype=torch.float32, device=dev) for _ in range(4))
    v = torch.empty((H, W), dtype=torch.uint8, device=dev)
    ws = torch.empty(lib.unw_workspace_bytes(H, W), dtype=torch.uint8, device=dev)
    _lib.check(lib.unw_setup_gradients(t.data_ptr(), None, H, W, gx.data_ptr(), gy.data_ptr(), wx.data_ptr(), wy.data_ptr(),
                                       v.data_ptr(), ws.data_ptr(), ws.numel(),
                                       ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)))
    g = gx.cpu().numpy()
    assert np.isnan(g[5, 6]) and np.isnan(g[5, 7])
    d = p[:, 1::2].astype(np.float64)
    got = g[:, 0:-1:2].astype(np.float64)
    ok = np.isfinite(d)
    ref = np.array([math.atan2(math.sin(x), math.cos(x)) for x in d[ok]])
    assert np.abs(got[ok]).max() <= float(np.float32(np.pi))
    e = np.abs(got[ok] - ref)
    assert np.minimum(e, np.abs(2 * np.pi - e)).max() <= tol
