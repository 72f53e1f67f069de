"""Row transforms of widths that are not powers of two, at the edges of each transform length.

A width W runs on Bluestein length M, the smallest of 2^k and 3 2^k that is at least 2 W - 1; the two forms of the
transform (ends in registers below M = 8192, through shared memory from there on unless M is three
times a power of two) and their zero padding are checked through the operator entry point at the
smallest and the largest width of each length, against the float64 operator with the bar of the other
preconditioner tests (2e-5 of the largest value).
"""
import numpy as np
import pytest
import scipy.fft as sfft

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from core_b200 import _lib  # noqa: E402

DEV = torch.device("cuda", 0)
LENGTHS = [256, 512, 768, 1024, 1536, 2048, 3072, 4096, 6144, 8192, 12288, 16384]
EDGES = sorted({w for lo, hi in zip([128] + LENGTHS, LENGTHS)
                for w in (lo // 2 + 1, hi // 2 - 1, hi // 2) if w & (w - 1)})


def operator64(r):
    H, W = r.shape
    lam = (4 * np.sin(np.pi * np.arange(H) / (2 * H)) ** 2)[:, None] + (4 * np.sin(np.pi * np.arange(W) / (2 * W)) ** 2)
    lam[0, 0] = 1.0
    t = sfft.dctn(r.astype(np.float64), type=2) / lam
    t[0, 0] = 0.0
    return sfft.idctn(t, type=2)


@pytest.mark.parametrize("W", EDGES)
@pytest.mark.parametrize("H", [1, 6])
def test_row_transform_at_the_edges_of_each_length(H, W):
    r = (np.random.default_rng(W).standard_normal((H, W)) + 0.5).astype(np.float32)
    lib = _lib.load()
    t = torch.from_numpy(r).to(DEV)
    z = torch.full((H, W), float("nan"), dtype=torch.float32, device=DEV)
    ws = torch.full((lib.unw_workspace_bytes(H, W),), 0xA5, dtype=torch.uint8, device=DEV)
    _lib.check(lib.unw_apply_preconditioner(t.data_ptr(), H, W, z.data_ptr(), ws.data_ptr(), ws.numel(),
                                            torch.cuda.current_stream(DEV).cuda_stream))
    z64 = operator64(r)
    assert np.abs(z.cpu().numpy() - z64).max() <= 2e-5 * np.abs(z64).max()
