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
