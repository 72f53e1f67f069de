"""IRLS iteration counts of converging solves are those of a float64 run (the float32 right-hand side, whose
rounding kept them iterating or ended them early, is not stored).  Scenes of the oracle whose rel_change stays at least 5% off
the stop tolerance in every iteration; the oracle's float32 run takes 7 and 3 iterations on the third and the last of them.
"""
import numpy as np
import pytest

from core_b200.synthetic import gen_g1
from oracle.irls_oracle import OracleStats, irls_unwrap_2d as oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import core_b200  # noqa: E402


@pytest.mark.parametrize("H,W,seed,weighted,iters", [(200, 180, 1, True, 3), (200, 180, 6, False, 2), (459, 687, 5, True, 4),
                                                     (256, 320, 3, False, 3), (512, 512, 7, False, 5)])
def test_counts_are_those_of_a_float64_run(H, W, seed, weighted, iters):
    p, c, _ = gen_g1(H, W, seed=seed)
    w = c if weighted else None
    ost = OracleStats()
    uo, _ = oracle(p, w, dtype=np.float64, stats=ost)
    assert ost.irls_iters == iters and all(abs(r / 1e-3 - 1) > 0.05 for r in ost.rel_change)
    u, _, st = core_b200.irls_unwrap_2d(p, w, return_stats=True)
    assert st["irls_iters"] == iters
    v = np.isfinite(p)
    e = (u[v].astype(np.float64) - uo[v])
    assert np.sqrt(np.mean((e - e.mean()) ** 2)) <= 1e-3
