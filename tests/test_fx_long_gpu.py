"""Accuracy of the long-series transforms (needs a GPU).

Frames of 4 x 4 whose zero wavevector is a multiple of 1/4: its structure function is known from integer sums.
The lags reach to 40 frames from the end, where the error of the correlation weighs most.  Yardstick: the error of
the float-float transforms that these replaced, over the same movies."""

import numpy as np
import pytest

from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("T,float_float", [(20000, 2.0e-13), (12000, 1.4e-13)])
def test_error_is_no_larger_than_in_float_float(built_lib, T, float_float):
    import fastddm_gb300 as fddm
    from scipy.signal import lfilter

    lags = sorted({int(v) for v in np.geomspace(1, T - 40, 25)})
    a = np.exp(-1.0 / 400)
    err = []
    for seed in range(32):
        rng = np.random.default_rng(seed)
        walk = lfilter([np.sqrt(1 - a * a)], [1, -a], rng.standard_normal(T))
        imgs = (2000 + 400 * walk[:, None, None] + 20 * rng.standard_normal((T, 4, 4))).round().clip(0, 65535)
        imgs = imgs.astype(np.uint16)
        got = fddm.ddm(imgs, lags, mode="fft")._data[:-2, 2, 0]
        f = imgs.sum(axis=(1, 2)).astype(np.int64)
        exact = np.array([float(((f[l:] - f[:T - l]) ** 2).sum()) / (16.0 * (T - l)) for l in lags])
        err.append(np.linalg.norm(got - exact) / np.linalg.norm(exact))
    assert np.sqrt(np.mean(np.square(err))) <= float_float


@pytest.mark.parametrize("split", [2, 4, 8])
@pytest.mark.parametrize("kind", ["one frequency", "one residue", "white"])
def test_pairs_of_unlike_power(built_lib, monkeypatch, split, kind):
    """Energy in one coefficient, in the coefficients of one residue (a series whose frames repeat), in all:
    the pairs' shifts differ most, or not at all.  Tolerance of test_fx_gpu.py, on the direct mode."""
    import fastddm_gb300 as fddm

    monkeypatch.setenv("FDDM_B200_TEMPORAL_SPLIT", str(split))
    T = 480
    t = np.arange(T)
    rng = np.random.default_rng(4)
    s = {"one frequency": np.cos(2 * np.pi * 5 * t / 960), "one residue": (t % 8 == 0) * 1.0,
         "white": rng.standard_normal(T)}[kind]
    imgs = (3000 + 300 * s[:, None, None] * rng.uniform(0.5, 1.0, (4, 6)) + rng.uniform(0, 2, (T, 4, 6))).astype(np.uint16)
    lags = [1, 2, 7, 8, 100, 240, 447, 460, 479]
    got = fddm.ddm(imgs, lags, mode="fft")._data
    ref = fddm.ddm(imgs, lags, mode="diff")._data
    rowmax = np.abs(ref).reshape(len(ref), -1).max(axis=1)[:, None, None]
    assert (np.abs(got - ref) <= 1e-8 * np.abs(ref) + 1e-13 * rowmax).all()


def test_power_in_one_coefficient(built_lib, monkeypatch):
    """A whole pair's power in one value, just below and above the powers of two that its shift is chosen by: the
    inverse passes double it, to just below 2^31."""
    import fastddm_gb300 as fddm

    monkeypatch.setenv("FDDM_B200_TEMPORAL_SPLIT", "8")
    T = 512
    tone = np.exp(2j * np.pi * 32 * np.arange(T) / 1024)
    # frames whose (0, 1) mode is the tone: two cosines along x, a quarter period apart
    x = np.exp(2j * np.pi * np.arange(8) / 8)
    lags = [1, 7, 64, 300, 470]
    for amplitude in np.linspace(1.0, 2.0, 33):
        imgs = (amplitude * (tone[:, None, None] * x[None, None, :]).real + np.zeros((T, 4, 8))).astype(np.float32)
        got = fddm.ddm(imgs, lags, mode="fft")._data[:-2, 2, 1]
        f = (imgs.astype(np.float64) * np.conj(x)[None, None, :]).sum(axis=(1, 2)) / np.sqrt(32.0)
        exact = np.array([np.mean(np.abs(f[l:] - f[:T - l]) ** 2) for l in lags])
        var = np.mean(np.abs(f - f.mean()) ** 2)
        assert (np.abs(got - exact) <= 16 * 2.0 ** -48 * var * T / (T - np.array(lags)) + 1e-13 * exact).all(), amplitude
