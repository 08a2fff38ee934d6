"""Batches whose many-job kernel needs shared memory about the 48 KB that a launch has without an opt-in (its
dynamic part and the kernel's static part count together), and groups of one job for every compiled length
(needs a GPU).  Results equal the single calls' bit for bit."""

import json
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from conftest import gpu_ready

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")]

ROOT = Path(__file__).resolve().parent.parent

# In a process of its own: a larger batch of the same kernel leaves the opt-in set.
CHILD = """
import json, sys
import numpy as np
import fastddm_gb300 as fddm
from fastddm_gb300 import autotune
from fastddm_gb300.batch import ddm_batch

tier, need, lengths = sys.argv[1], int(sys.argv[2]), json.loads(sys.argv[3])
bad = {}
for T in lengths:
    autotune.set_entry(tier, "fft", T, T - 1, 128, need)
    frames = np.random.default_rng(T).integers(0, 4000, (T, 6, 10)).astype(np.uint16)
    try:
        got = ddm_batch([frames], range(1, T), precision=tier)[0]._data
    except RuntimeError as e:
        bad[T] = str(e)
        continue
    if not np.array_equal(got, fddm.ddm(frames, range(1, T), mode="fft", precision=tier)._data):
        bad[T] = "differs"
print(json.dumps(bad))
"""


# dynamic sizes just below 48 KB, where the static part decides: first, middle and last length of each range
# (every lag, 128 threads, tables in global scratch or in shared memory), and the neighbours outside
@pytest.mark.parametrize("tier,need,lengths", [
    ("ff", 0, [1152, 1153, 1253, 1267, 1277, 1280, 1296, 1297]), ("ff", 1, [559, 560, 576, 577]),
    ("f64", 0, [1152, 1153, 1277, 1296]), ("f64", 1, [560, 576]),
    ("f32", 0, [2231, 2232, 2270, 2304]), ("f32", 1, [800, 825, 851]),
])
def test_batches_near_48_kilobytes(built_lib, tier, need, lengths):
    r = subprocess.run([sys.executable, "-c", CHILD, tier, str(need), json.dumps(lengths)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert json.loads(r.stdout.strip().splitlines()[-1]) == {}


def test_every_compiled_length_in_one_batch(built_lib):
    """2 x 2^6 .. 2 x 2^12 points and a general plan: groups of one job each."""
    import fastddm_gb300 as fddm
    from fastddm_gb300.batch import ddm_batch

    rng = np.random.default_rng(1)
    stacks = [rng.integers(0, 4000, (T, 5, 8)).astype(np.uint16) for T in (64, 128, 256, 512, 1024, 2048, 4096, 343)]
    lags = [[1, 2, s.shape[0] // 2, s.shape[0] - 1] for s in stacks]
    for s, lg, r in zip(stacks, lags, ddm_batch(stacks, lags)):
        np.testing.assert_array_equal(r._data, fddm.ddm(s, lg, mode="fft")._data)
