"""The diff kernel's groups of one, two and four lags a warp (needs a GPU): numbers of lags about once and twice the
warps of every CTA size, series about the length where groups of four are always taken, lags down to one pair.
Yardstick and tolerance as in test_ddm_gpu.py."""

import numpy as np
import pytest

import ddm_oracle as oracle
from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("T", [255, 256, 700])
@pytest.mark.parametrize("share", [1, 2])
def test_group_sizes(built_lib, monkeypatch, threads, T, share):
    import fastddm_gb300 as fddm

    monkeypatch.setenv("FDDM_B200_TEMPORAL_THREADS", str(threads))
    rng = np.random.default_rng(T)
    imgs = (1000 + 20 * np.cumsum(rng.standard_normal((T, 3, 4)), axis=0)).clip(0, 65535).astype(np.uint16)
    warps = threads // 32
    for nlags in sorted({1, share * warps - 1, share * warps, share * warps + 1}):
        lags = sorted({int(v) for v in np.linspace(1, T - 1, nlags)}) if nlags > 1 else [T - 1]
        assert len(lags) == nlags
        got = fddm.ddm(imgs, lags, mode="diff")._data
        ex = oracle.ddm_exact(imgs, oracle.prepare_lags(lags, T), 4, 3)
        rowmax = np.abs(ex).reshape(ex.shape[0], -1).max(axis=1)[:, None, None]
        assert (np.abs(got - ex) <= 1e-8 * np.abs(ex) + 1e-13 * rowmax).all(), nlags
