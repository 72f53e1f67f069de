"""Goldstein adaptive filter (insardev/insardev/utils_goldstein.py:157-330, the GPU path).

Golden fixtures: the reference's own goldstein_pytorch run on the CPU torch
device (tests/golden/make_goldstein_golden.py).  CPU tests pin the oracle to
them; GPU tests compare the CUDA filter with the fixtures and the oracle.
Tolerance: NaN positions identical; max |out - ref| <= 2e-5 * max |ref|
(float32 FFTs of different association orders).
"""
import ctypes as C
import glob
import os

import numpy as np
import pytest

from conftest import REPO
from oracle.goldstein_oracle import goldstein as oracle_goldstein

GOLD = sorted(glob.glob(os.path.join(REPO, "tests", "golden", "gs_*.npz")))


def _load(path):
    d = np.load(path)
    py, px = (int(v) for v in d["psize"])
    return d["phase"], d["corr"], py, px, float(d["threshold"]), d["out"]


def _close(out, ref, tol):
    nm = np.isnan(ref)
    assert (np.isnan(out) == nm).all()
    if (~nm).any():
        err = np.abs(out[~nm] - ref[~nm]).max() / np.abs(ref[~nm]).max()
        assert err <= tol, err


def test_fixtures_present():
    assert len(GOLD) >= 5


@pytest.mark.parametrize("path", GOLD, ids=[os.path.basename(p)[:-4] for p in GOLD])
def test_oracle_matches_reference_fixture(path):
    z, corr, py, px, thr, ref = _load(path)
    _close(oracle_goldstein(z, corr, py, px, thr), ref, 2e-6)


def test_goldstein_rejects_bad_args_without_gpu():
    from core_b200 import _lib
    lib = _lib.load()
    assert lib.unw_goldstein_workspace_bytes(64, 64, 32, 32) > 64 * 64 * 12
    assert lib.unw_goldstein_workspace_bytes(64, 64, 24, 32) == 0
    assert lib.unw_goldstein_workspace_bytes(64, 64, 128, 32) == 0
    f = C.c_void_p(0x10000)
    rc = lib.unw_goldstein_c64(None, 8, f, 8, 8, 8, 4, 4, 0.5, f, 8, f, 1 << 30, None)
    assert rc == _lib.UNW_E_ARG
    rc = lib.unw_goldstein_c64(f, 8, f, 8, 8, 8, 6, 4, 0.5, f, 8, f, 1 << 30, None)
    assert rc == _lib.UNW_E_UNSUPPORTED
    rc = lib.unw_goldstein_c64(f, 8, f, 8, 8, 8, 4, 4, 1.5, f, 8, f, 1 << 30, None)
    assert rc == _lib.UNW_E_ARG
    rc = lib.unw_goldstein_c64(f, 8, f, 8, 8, 8, 4, 4, 0.5, f, 8, f, 16, None)
    assert rc == _lib.UNW_E_WORKSPACE


# ------------------------------------------------------------------ GPU
def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.gpu
@pytest.mark.parametrize("path", GOLD, ids=[os.path.basename(p)[:-4] for p in GOLD])
def test_cuda_matches_reference_fixture(path):
    _gpu()
    import core_b200
    z, corr, py, px, thr, ref = _load(path)
    out = core_b200.goldstein(z, corr, py, px, threshold=thr)
    assert out.dtype == np.complex64 and out.shape == z.shape
    _close(out, ref, 2e-5)


@pytest.mark.gpu
def test_cuda_matches_oracle_larger_and_tensor_io():
    torch = _gpu()
    import core_b200
    from core_b200.synthetic import gen_g1
    p, c, _ = gen_g1(300, 257, seed=9, noise=0.7)
    z = np.exp(1j * p.astype(np.float64)).astype(np.complex64)
    z[np.isnan(p)] = np.nan
    ref = oracle_goldstein(z, c, 32, 32, 0.5)
    out = core_b200.goldstein(z, c, {"y": 32, "x": 32})
    _close(out, ref, 2e-5)
    dev = torch.device("cuda", 0)
    t = core_b200.goldstein(torch.from_numpy(z).to(dev), torch.from_numpy(c).to(dev), 32)
    assert t.is_cuda and t.dtype == torch.complex64
    np.testing.assert_array_equal(t.cpu().numpy(), out)   # deterministic


# patch sizes and grids at which the walk changes form: every patch size, unequal sides, grids smaller
# than a patch, one row or column, cells that end at the edge of a CTA's strip or walk, and patches that
# are not valid; 2e-5 of the largest value as above
@pytest.mark.gpu
@pytest.mark.parametrize("shape,py,px,thr", [((300, 257), 4, 4, 0.5), ((130, 251), 8, 8, 0.5), ((97, 483), 16, 16, 0.5),
                                             ((65, 225), 32, 32, 0.5), ((200, 193), 64, 64, 0.3), ((90, 300), 64, 4, 0.5),
                                             ((70, 290), 4, 64, 0.5), ((33, 40), 32, 16, 0.5), ((129, 50), 8, 32, 0.7),
                                             ((100, 200), 16, 64, 0.5), ((80, 99), 64, 32, 0.5), ((5, 7), 32, 32, 0.0),
                                             ((1, 300), 16, 16, 0.02), ((300, 1), 32, 8, 0.01), ((16, 16), 16, 16, 1.0)])
def test_cuda_matches_oracle_at_the_edges(shape, py, px, thr):
    _gpu()
    import core_b200
    rng = np.random.default_rng(py * 1000 + px + shape[0])
    z = (np.exp(1j * rng.uniform(-3, 3, shape)) * rng.uniform(0.2, 5, shape)).astype(np.complex64)
    z[rng.random(shape) < 0.1] = np.nan
    z[: shape[0] // 3, : shape[1] // 4] = np.nan
    corr = rng.uniform(0, 1, shape).astype(np.float32)
    corr[rng.random(shape) < 0.05] = np.nan
    ref = oracle_goldstein(z, corr, py, px, thr, dtype=np.float64)
    out = core_b200.goldstein(z, corr, py, px, threshold=thr)
    nm = np.isnan(ref)
    assert (np.isnan(out) == nm).all()
    if (~nm).any():   # a single row or column has zero taper: all zeros, exactly
        assert np.abs(out[~nm] - ref[~nm]).max() <= 2e-5 * np.abs(ref[~nm]).max()


@pytest.mark.gpu
def test_cuda_result_in_place_of_the_input():
    torch = _gpu()
    import core_b200
    from core_b200 import _lib
    rng = np.random.default_rng(5)
    z = np.exp(1j * rng.uniform(-3, 3, (150, 170))).astype(np.complex64)
    corr = rng.uniform(0, 1, z.shape).astype(np.float32)
    ref = core_b200.goldstein(z, corr, 16)
    dev = torch.device("cuda", 0)
    t, c = torch.from_numpy(z).to(dev), torch.from_numpy(corr).to(dev)
    lib = _lib.load()
    ws = torch.empty(lib.unw_goldstein_workspace_bytes(150, 170, 16, 16), dtype=torch.uint8, device=dev)
    _lib.check(lib.unw_goldstein_c64(t.data_ptr(), 170, c.data_ptr(), 170, 150, 170, 16, 16, 0.5, t.data_ptr(), 170,
                                     ws.data_ptr(), ws.numel(), torch.cuda.current_stream(dev).cuda_stream))
    np.testing.assert_array_equal(t.cpu().numpy(), ref)


def _impulses(shape, amplitude):
    """Real impulses in the middle of every second 8 x 8 cell block: each 8 x 8 patch of the interior holds
    at most one, so its spectrum has the same modulus everywhere."""
    z = np.zeros(shape, np.complex64)
    z[6::16, 6::16] = amplitude
    return z


# Coherence 0 makes the power 1: the spectrum of an impulse A becomes A |A| everywhere, and its inverse sum
# 64 A |A| passes float32 in the last butterfly alone (32 A |A| is below 3.4e38).  The sum is divided by the
# number of patches as any other: an infinite sum stays infinite, and nothing turns into NaN.
@pytest.mark.gpu
def test_cuda_overflowed_sum_stays_infinite():
    _gpu()
    import core_b200
    z = _impulses((48, 64), np.float32(2.5e18))
    out = core_b200.goldstein(z, np.zeros(z.shape, np.float32), 8, 8, 0.5)
    at = z != 0
    assert np.isposinf(out.real[at]).all() and np.isfinite(out.imag[at]).all()
    assert np.isfinite(out[~at]).all()


# The spectrum weight max(|F|, 1e-10)^alpha by itself, against the float64 power: an impulse A of weight 1 in its
# patches comes out as A max(A, 1e-10)^alpha times the mean of the four tapers over it.  Coherence c (constant)
# gives alpha = 1 - c, outside [0, 1] too, |alpha| <= 2 and beyond (where the general form runs), and A goes from
# below the floor of 1e-10 to moduli whose square is beyond float32.  Relative tolerance, from the
# operations' bounds: 4e-6 for twelve butterfly stages (3.8 u each, u = 2^-24) and the power itself, and 8e-7 |c|
# for alpha (11 additions of the weighted coherence and two roundings) times |ln A|, which the power multiplies it by.
# Pairs whose weighted spectrum, or its sum, is outside float32 are left out.
COHERENCES = [0.0, 0.5, 1.0, 0.96875, -0.75, -1.0, 1.75, 3.0, -1.5, 4.5]
AMPLITUDES = [3e-12, 1e-10, 7.3e-8, 1e-4, 0.711, 1.0, 1.413, 37.0, 1e6, 2.2e12, 3.1e18, 4.7e18, 1.6e19, 1.9e19, 1e20, 2.5e24]


@pytest.mark.gpu
@pytest.mark.parametrize("c,amp", [(c, a) for c in COHERENCES for a in AMPLITUDES if 9e-31 < a * max(a, 1e-10) ** (1 - c) < 1e36])
def test_cuda_spectrum_weight_of_an_impulse(c, amp):
    _gpu()
    import core_b200
    z = _impulses((48, 64), np.float32(amp))
    A = float(np.float32(amp))
    held = A * float(np.float32(max(A, 1e-10) ** (1.0 - c)))   # the power is a float32 (zero below 1e-45)
    out = core_b200.goldstein(z, np.full(z.shape, c, np.float32), 8, 8, 0.5)
    taper = 1.0 - abs(np.array([2.0, 1.0]) - 3.0) / 3.0   # local rows 2 and 6 (mirrored: 1)
    ref = held * np.outer(taper, taper).sum() / 4
    # impulses whose four patches lie inside the grid (beyond it the coherence is 0)
    at = [(y, x) for y in (6, 22, 38) for x in (6, 22, 38, 54)]
    got = np.array([out[p] for p in at])
    tol = 4e-6 + 8e-7 * abs(c) * abs(np.log(A))
    assert np.abs(got - ref).max() <= tol * ref
