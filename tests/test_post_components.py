"""Components of the valid mask at the borders of the row pieces that the post-processing walks.

The labels start from runs of valid pixels within 512-column pieces of a row and are joined across
piece borders and with the row below at the first pixel of a pair of overlapping runs.  Masks
with runs that end, start or pass at the 32- and 512-column borders, combs, spirals and noise are
compared with scipy's labelling through a solve (component sizes and partition).
"""
import numpy as np
import pytest
from scipy import ndimage as ndi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import core_b200  # noqa: E402


def _masks():
    rng = np.random.default_rng(3)
    comb = np.zeros((40, 1100), bool)
    comb[0] = True
    comb[:, ::2] = True
    comb[20, :] = False
    snake = np.ones((33, 700), bool)
    snake[1::4, :-1] = False
    snake[3::4, 1:] = False
    borders = np.ones((50, 1540), bool)
    borders[:, [31, 32, 511, 512, 1023, 1024, 1535]] = False
    borders[7, [31, 511, 1024]] = True
    borders[30, [32, 512]] = True
    noise = rng.random((90, 601)) < 0.6
    dots = np.zeros((20, 1030), bool)
    dots[::2, ::3] = True
    return {"comb": comb, "snake": snake, "borders": borders, "noise": noise, "dots": dots,
            "column": np.ones((700, 1), bool), "row": np.ones((1, 1300), bool)}


@pytest.mark.parametrize("name", sorted(_masks()))
def test_components_match_scipy_labels(name):
    m = _masks()[name]
    yy, xx = np.mgrid[:m.shape[0], :m.shape[1]]
    p = np.where(m, np.angle(np.exp(1j * (0.05 * xx - 0.03 * yy))), np.nan).astype(np.float32)
    _, cc = core_b200.irls_unwrap_2d(p, max_iter=1, cg_max_iter=2, conncomp_size=1)
    lab, n = ndi.label(m)
    assert (cc > 0).sum() == m.sum() and cc.max() == n
    pairs = np.unique(np.stack([lab[m], cc[m].astype(np.int64)]), axis=1)
    assert pairs.shape[1] == n                      # one label per component, and no two share one
    sizes = np.bincount(cc[m].astype(np.int64))[1:]
    assert (np.diff(sizes) <= 0).all()
