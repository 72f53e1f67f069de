"""The column half of the DCT preconditioner as a tridiagonal solve per column (unw_col_tri.cu).

Checked through the operator entry point against the float64 operator idct2(dct2(r) / lambda), with
the bar of the other preconditioner tests (2e-5 of the largest value: the rows still go
through float32 transforms), at the sizes where the pass changes form: columns shorter than
the 64- and 32-row halos, one row, the edges of the 128- / 192-row tiles (test_column_pass_edges.py has
those of the 384- / 448-row ones, which larger grids take), strips that end inside 64 columns, grids of wide columns only, odd widths (no 8-byte pairs), the longest column.
The solver is checked against the float64 oracle: float32 only enters in the stored vectors, so the
result is float32-close to it.
"""
import numpy as np
import pytest
import scipy.fft as sfft

from core_b200.synthetic import gen_g1
from oracle.irls_oracle import irls_unwrap_2d as oracle_unwrap

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import core_b200  # noqa: E402
from core_b200 import _lib  # noqa: E402

DEV = torch.device("cuda", 0)


def operator64(r):
    H, W = r.shape
    lam = (4 * np.sin(np.pi * np.arange(H) / (2 * H)) ** 2)[:, None] + (4 * np.sin(np.pi * np.arange(W) / (2 * W)) ** 2)
    lam[0, 0] = 1.0
    t = sfft.dct(sfft.dct(r.astype(np.float64), type=2, axis=1), type=2, axis=0) / lam
    t[0, 0] = 0.0
    return sfft.idct(sfft.idct(t, type=2, axis=0), type=2, axis=1)


@pytest.mark.parametrize("shape", [(1, 64), (2, 65), (1, 1000), (31, 100), (33, 257), (63, 500), (64, 363), (65, 700),
                                   (127, 130), (129, 131), (191, 1000), (193, 1001), (1025, 90), (385, 3000),
                                   (449, 2999), (4099, 1400), (300, 33), (300, 32), (97, 5), (13000, 8), (28672, 3)])
def test_column_pass_matches_float64_operator(shape):
    rng = np.random.default_rng(shape[0] * 8191 + shape[1])
    r = (rng.standard_normal(shape) + 0.5).astype(np.float32)     # a mean, which the operator drops
    H, W = shape
    lib = _lib.load()
    t = torch.from_numpy(r).to(DEV)
    z = torch.full((H, W), float("nan"), dtype=torch.float32, device=DEV)
    ws = torch.full((lib.unw_workspace_bytes(H, W),), 0xA5, dtype=torch.uint8, device=DEV)
    _lib.check(lib.unw_apply_preconditioner(t.data_ptr(), H, W, z.data_ptr(), ws.data_ptr(), ws.numel(),
                                            torch.cuda.current_stream(DEV).cuda_stream))
    z64 = operator64(r)
    assert np.abs(z.cpu().numpy() - z64).max() <= 2e-5 * max(np.abs(z64).max(), 1e-30)


@pytest.mark.parametrize("shape", [(150, 211), (256, 320)])
def test_solve_is_float32_close_to_the_float64_oracle(shape):
    # float32 output and PCG correction: a few ulps of the largest value (|u| < 64: ulp 3.8e-6)
    p, c, _ = gen_g1(*shape, seed=31)
    u, _ = core_b200.irls_unwrap_2d(p, c)
    uo, _ = oracle_unwrap(p, c, dtype=np.float64)
    v = np.isfinite(p)
    assert np.abs(uo[v]).max() < 64
    assert np.sqrt(np.mean((u[v].astype(np.float64) - uo[v]) ** 2)) <= 4 * 3.8e-6
