"""Series whose lags are all direct sums, about the line of 32 pairs of frames, where the fixed-point temporal
kernel runs no transform (needs a GPU).  Yardstick and tolerance as in test_ddm_gpu.py."""

import numpy as np
import pytest

import ddm_oracle as oracle
from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]


# all lags direct, one not, only late ones; compile-time lengths and general ones; more modes than CTAs
@pytest.mark.parametrize("T,first,shape", [
    (2, 1, (40, 64)), (3, 1, (5, 6)), (16, 1, (40, 64)), (32, 1, (40, 64)), (33, 1, (40, 64)), (34, 1, (40, 64)),
    (34, 2, (5, 6)), (40, 8, (5, 6)), (40, 7, (5, 6)), (343, 311, (5, 6)), (343, 310, (5, 6)), (512, 490, (5, 6)),
])
def test_direct_lags(built_lib, T, first, shape):
    import fastddm_gb300 as fddm

    rng = np.random.default_rng(T)
    imgs = (1000 + 30 * np.cumsum(rng.standard_normal((T, *shape)), axis=0)).clip(0, 65535).astype(np.uint16)
    lags = list(range(first, T))
    got = fddm.ddm(imgs, lags, mode="fft")._data
    nx, ny = oracle.next_fast_len_cpp(shape[1]), oracle.next_fast_len_cpp(shape[0])
    ex = oracle.ddm_exact(imgs, oracle.prepare_lags(lags, T), nx, ny)
    rowmax = np.abs(ex).reshape(ex.shape[0], -1).max(axis=1)[:, None, None]
    assert (np.abs(got - ex) <= 1e-8 * np.abs(ex) + 1e-13 * rowmax).all()
