"""The azimuthal average's bins made on the device against the host's, bit for bit (every sum adds in pixel
order on both), and the rule that chooses between them."""

import numpy as np
import pytest

from conftest import gpu_ready


def _case(n, bins, form, seed):
    rng = np.random.default_rng(seed)
    dist = rng.uniform(0.0, 10.0, (1, n))
    mask = weights = counts = rng_ = None
    if form == "masked":
        mask = rng.random((1, n)) < 0.6
    elif form == "weighted":
        weights = rng.uniform(0.0, 2.0, (1, n)) * (rng.random((1, n)) < 0.7)
        counts = rng.integers(0, 3, (1, n))
    elif form == "ties":  # distances on the edges, edges twice, a bound above the first edges
        dist = np.round(dist)
        bins = np.sort(np.concatenate([np.arange(bins), np.arange(0, bins, 3)])).astype(float)
        rng_ = (2.0, 7.0)
    elif form == "nonfinite":
        dist[0, ::5], dist[0, 1::7], dist[0, 2::11] = np.nan, np.inf, -np.inf
        rng_ = (0.5, 9.0)
    return dist, bins, rng_, mask, weights, counts


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("form", ["plain", "masked", "weighted", "ties", "nonfinite"])
@pytest.mark.parametrize("n,bins", [(1, 1), (31, 2), (33, 33), (1023, 5), (1024, 32), (1025, 600), (9000, 31), (70001, 16384)])
def test_device_bins(built_lib, n, bins, form):
    import torch

    from fastddm_gb300 import azimuthalaverage as az

    dist, edges, rng_, mask, weights, counts = _case(n, bins if form != "ties" else min(bins, 4096), form, n + bins)
    device = torch.device("cuda", 0)
    args = az.bin_arguments(dist, edges, rng_, mask, weights, counts, True)
    got = az._bins_on_device(dist, args, device)
    setup = az.bin_sums(dist, args)
    want = az._upload_bins(setup, True, device)
    total = int(want.offsets[-1])
    assert torch.equal(got.offsets, want.offsets)
    assert torch.equal(got.pixels[:total], want.pixels[:total])
    np.testing.assert_array_equal(got.sum_wi.cpu().numpy(), want.sum_wi.cpu().numpy())
    np.testing.assert_array_equal(got.bias.cpu().numpy(), want.bias.cpu().numpy())
    k = got.mean.cpu().numpy()
    az._fill_empty(k, setup.sum_wi, args.bin_edges)
    np.testing.assert_array_equal(k, setup.k)


@pytest.mark.parametrize("what,usable", [
    ("plain", True), ("list", True), ("integers", True), ("small", False), ("float32", False), ("swapped", False),
    ("unordered list", False), ("infinite edge", False), ("nan distance", True), ("nan edges", False), ("masked array", False),
])
def test_rule(what, usable):
    from fastddm_gb300 import azimuthalaverage as az

    dist = np.random.default_rng(0).uniform(0.0, 9.0, (128, 128))
    bins = np.linspace(0.0, 9.0, 20)
    if what == "list":
        bins = bins.tolist()
    elif what == "integers":
        bins = np.arange(10)
    elif what == "small":
        dist = dist[:1, :3]
    elif what == "float32":
        dist = dist.astype(np.float32)
    elif what == "swapped":
        dist = dist.astype(">f8")
    elif what == "unordered list":
        bins = [1.0, 3.0, 2.0]  # lists compare in lexicographic order
    elif what == "infinite edge":
        bins = [0.0, 3.0, np.inf]
    elif what == "nan distance":
        dist[3, 4] = np.nan
    elif what == "nan edges":
        dist[3, 4] = np.nan
        bins = 12
    elif what == "masked array":
        dist = np.ma.masked_less(dist, 1.0)
    args = az.bin_arguments(dist, bins, None, None, None, None, True)
    assert az._device_bins_usable(dist, args) is usable


@pytest.mark.parametrize("shape,bins,weighted,usable", [
    ((513, 1024), 2, False, False), ((513, 1024), 3, False, False), ((513, 1024), 5, False, False),
    ((513, 1024), 20, False, True), ((513, 1024), 512, True, True), ((513, 1024), 5, True, False),
    ((65, 128), 10, False, False), ((65, 128), 40, False, True), ((129, 129), 2, False, False),
])
def test_bins_that_hold_most_pixels_stay_on_the_host(shape, bins, weighted, usable):
    """A bin's sums are one chain of additions: a map that falls into one or two bins is slower on the device."""
    from fastddm_gb300 import azimuthalaverage as az

    ky, kx = np.arange(shape[1]) - shape[1] // 2, np.arange(shape[0])
    dist = np.hypot(*np.meshgrid(kx, ky)) / shape[0]
    w = np.random.default_rng(0).uniform(0.0, 1.0, dist.shape) if weighted else None
    args = az.bin_arguments(dist, bins, None, None, w, None, True)
    assert az._device_bins_usable(dist, args) is usable
    # a mask that leaves one pixel in fifty shortens the lists
    mask = np.random.default_rng(1).random(dist.shape) < 0.02
    args = az.bin_arguments(dist, bins, None, mask, w, None, True)
    assert az._device_bins_usable(dist, args) is True


@pytest.mark.parametrize("npix", [1, 4096, 525312, 4096 * 2049, 30000 * 20000])
@pytest.mark.parametrize("bins", [1, 513, 16384])
def test_scratch_is_bounded(npix, bins):
    """The chunk table stays within the pixels' own size or 16 MB."""
    import ctypes

    from fastddm_gb300 import _build, _lib

    _build.build()
    need = ctypes.c_size_t()
    _lib.check(_lib.load().fddm_b200_azimuthal_bins_workspace(npix, bins, ctypes.byref(need)))
    assert 4 * npix < need.value <= 4 * npix + max(4 * npix, 1 << 24)


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_ready(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("form", ["plain", "masked"])
@pytest.mark.parametrize("n,bins", [(262145, 16384), (300001, 16384), (1100000, 16384), (1100000, 9000)])
def test_longer_chunks(built_lib, n, bins, form):
    """Chunks of more than 1024 pixels (2048 and up), ragged last ones among them."""
    test_device_bins(built_lib, n, bins, form)


def test_host_setup_where_device_memory_runs_out(monkeypatch):
    torch = pytest.importorskip("torch")
    from fastddm_gb300 import azimuthalaverage as az

    def full(*_):
        raise torch.OutOfMemoryError("CUDA out of memory")

    monkeypatch.setattr(az, "_bins_on_device", full)
    dist, edges, rng_, mask, weights, counts = _case(9000, 40, "masked", 0)
    args = az.bin_arguments(dist, edges, rng_, mask, weights, counts, True)
    assert az._device_bins_usable(dist, args)
    tables, setup = az._bin_tables(dist, args, True, torch.device("cpu"))
    np.testing.assert_array_equal(tables.sum_wi.numpy(), setup.sum_wi)
    assert int(tables.offsets[-1]) == int(setup.valid.sum())
