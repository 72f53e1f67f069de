"""The captured graph of five PCG iterations: caps that it does not divide, and caps below its use.

The graph serves solves with at least ten PCG iterations; what is left over a multiple of five goes launch by
launch.  All kernels are deterministic, so a solve gives the same bits as with direct launches only.
"""
import ctypes as C

import numpy as np
import pytest

from core_b200.synthetic import gen_g2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from core_b200 import _lib  # noqa: E402
from core_b200.irls import make_params  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("cg", [1, 4, 9, 10, 11, 14, 15, 23])
def test_caps_that_the_graph_does_not_divide(cg, fixed):
    H, W = 150, 211
    p, c, _ = gen_g2(H, W, seed=19)
    ph, wt = (torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV) for a in (p, c))
    lib = _lib.load()
    ws = torch.empty(lib.unw_workspace_bytes(H, W), dtype=torch.uint8, device=DEV)
    out = []
    for flag in (0, _lib.UNW_F_NO_GRAPH):
        prm = make_params(max_iter=3, cg_max_iter=cg, fixed_iters=fixed)
        prm.flags |= flag
        u = torch.empty((H, W), dtype=torch.float32, device=DEV)
        cc = torch.empty((H, W), dtype=torch.int16, device=DEV)
        st = _lib.UnwStats()
        _lib.check(lib.unw_solve_f32(ph.data_ptr(), W, wt.data_ptr(), W, H, W, C.byref(prm), u.data_ptr(), W, cc.data_ptr(), W,
                                     ws.data_ptr(), ws.numel(), C.byref(st), torch.cuda.current_stream(DEV).cuda_stream))
        d = st.as_dict()
        if fixed:
            assert d["irls_iters"] == 3 and d["cg_iters_total"] == 3 * cg
        out.append((u.cpu().numpy().view(np.uint32), cc.cpu().numpy(), d["irls_iters"], d["cg_iters_total"]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][2:] == out[1][2:]
