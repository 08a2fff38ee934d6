"""The strongest cancellation of the temporal stage (needs a GPU): series that alternate from frame to frame, whose
structure function at even lags is millions of times below the variance.

Tolerance: the fixed-point transforms round at about 2^-48 of a mode's variance (tests/test_fx_gpu.py), sixteen of
which are allowed for the passes and the sums, times T / (T - lag) for the lag's normalisation; and 1e-13 of the
value for the spatial transforms."""

import numpy as np
import pytest

import ddm_oracle as oracle
from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("T", [500, 1024, 4000, 6000, 12000])
def test_alternating_frames(built_lib, T):
    import fastddm_gb300 as fddm

    rng = np.random.default_rng(3)
    sign = np.where(np.arange(T) % 2, -1.0, 1.0)
    imgs = (2000 + 500 * sign[:, None, None] * rng.standard_normal((4, 6)) + rng.standard_normal((T, 4, 6))).round()
    imgs = imgs.astype(np.uint16)
    lags = sorted({1, 2, 3, 4, 10, 100, T // 4, T // 2, T - 41, T - 40, T - 2, T - 1})
    got = fddm.ddm(imgs, lags, mode="fft")._data
    ex = oracle.ddm_exact(imgs, oracle.prepare_lags(lags, T), 6, 4)
    var = ex[-1]
    for l, g, e in zip(lags, got, ex):
        assert (np.abs(g - e) <= 16 * 2.0 ** -48 * var * T / (T - l) + 1e-13 * np.abs(e)).all(), l
