"""The diff kernel on series whose frames differ by many orders of magnitude (needs a GPU): lags that meet none of
the bright frames, which set the mode's fixed-point unit, keep the precision of float-float differences.

Yardstick: FP64 transforms of every frame and direct differences.  Tolerance: float-float carries 2^-48 of a
sample; a dozen roundings of that size per transform and difference, and the differences of a few pairs being up
to four times smaller than the samples, give 2^-43 of a lag's 2-norm over the modes."""

import numpy as np
import pytest

from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("T", [60, 600, 4000, 9000])
@pytest.mark.parametrize("form", ["frame", "first", "block", "ramp", "plain"])
@pytest.mark.parametrize("bits", [8, 16, 24])
def test_bright_frames(built_lib, T, form, bits):
    import fastddm_gb300 as fddm

    rng = np.random.default_rng(T + bits)
    imgs = 1.0 + 0.1 * rng.standard_normal((T, 8, 8))
    if form == "frame":
        imgs[T // 2] *= 2.0 ** bits
    elif form == "first":
        imgs[0] *= 2.0 ** bits
    elif form == "block":
        imgs[3 * T // 8: 5 * T // 8] *= 2.0 ** bits
    elif form == "ramp":
        imgs *= 2.0 ** np.linspace(0, bits, T)[:, None, None]
    imgs = imgs.astype(np.float32)
    lags = sorted({1, 2, T // 4, T // 2 + 1, 5 * T // 8 + 1, 3 * T // 4, T - 40, T - 5, T - 1})
    got = fddm.ddm(imgs, lags, mode="diff")._data[:-2]
    f = np.fft.fftshift(np.fft.rfft2(imgs.astype(np.float64)) / 8.0, axes=1)
    for l, g in zip(lags, got):
        exact = (np.abs(f[l:] - f[:T - l]) ** 2).mean(axis=0)
        assert np.linalg.norm(g - exact) <= 2.0 ** -43 * np.linalg.norm(exact), l


# the sum of squares about the mean just below, just above and well above the largest FP32 number
@pytest.mark.parametrize("largest", [3.37e38, 3.5e38, 1e39])
def test_energy_beyond_fp32(built_lib, largest):
    """Finite frames whose energy does not fit in FP32 keep their lags, power spectrum and variance."""
    import fastddm_gb300 as fddm

    rng = np.random.default_rng(0)
    T = 33
    base = rng.standard_normal((T, 1, 1)) + np.zeros((T, 4, 4))
    scale = np.sqrt(largest / (16.0 * ((base[:, 0, 0] - base[:, 0, 0].mean()) ** 2).sum()))
    imgs = (base * scale).astype(np.float32)
    got = fddm.ddm(imgs, [1, 20, 30], mode="diff")._data[:, 2, 0]
    f = imgs.astype(np.float64).sum(axis=(1, 2)) / 4.0
    exact = [((f[l:] - f[:T - l]) ** 2).mean() for l in (1, 20, 30)] + [(f ** 2).mean(), ((f - f.mean()) ** 2).mean()]
    for g, e, pairs in zip(got, exact, (32, 13, 3, 0, 0)):
        if pairs == 0 or e * pairs < 3e38:  # a lag's own sum is a float-float one
            assert abs(g - e) <= 1e-12 * e
