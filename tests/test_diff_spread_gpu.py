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
