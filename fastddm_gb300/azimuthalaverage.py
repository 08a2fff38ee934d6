"""Azimuthal average of the image structure function on the GB300.

Interface of the reference's ``src/python/azimuthalaverage.py``:
``AzimuthalAverage`` (``:80-274``), ``azimuthal_average_array`` (``:277-478``)
and ``azimuthal_average`` (``:481-564``).

Work split:

* host: argument checks, bin edges (``linspace`` edges, not ``bins + 1``), the
  weight of every pixel;
* device (``fddm_b200_azimuthal_bins``; numpy for small maps and what the device
  search does not take): bin indices, the mask (out-of-range, below ``x_min``,
  masked, zero weight), every bin's pixels in order, per-bin sums of weights
  and the weighted mean ``k`` per bin.  Both add in pixel order, the order of
  the reference's loops, so these match it bit for bit;
* device (``fddm_b200_azimuthal_average``, O(pixels x rows)): the weighted mean
  and unbiased weighted standard deviation of every row in every bin, one
  thread per (bin, row) summing in pixel order with the reference's operation
  order, so they also match the reference's loops bit for bit.
"""

from __future__ import annotations

import ctypes
import warnings
from dataclasses import dataclass
from typing import Iterable, Optional, Tuple, Union

import numpy as np

from . import _lib
from ._config import DTYPE
from .imagestructurefunction import ImageStructureFunction

try:
    import torch
except ImportError:  # pragma: no cover
    torch = None


@dataclass
class AzimuthalAverage:
    """Azimuthal average container (same fields as the reference)."""

    _data: np.ndarray
    _err: Optional[np.ndarray]
    k: np.ndarray
    tau: np.ndarray
    bin_edges: np.ndarray

    @property
    def data(self) -> np.ndarray:
        return self._data[:, :-2]

    @property
    def err(self) -> Optional[np.ndarray]:
        return None if self._err is None else self._err[:, :-2]

    @property
    def power_spec(self) -> np.ndarray:
        return self._data[:, -2]

    @property
    def var(self) -> np.ndarray:
        return self._data[:, -1]

    @property
    def power_spec_err(self) -> Optional[np.ndarray]:
        return None if self._err is None else self._err[:, -2]

    @property
    def var_err(self) -> Optional[np.ndarray]:
        return None if self._err is None else self._err[:, -1]

    def save(self, fname: str = "analysis_blob") -> None:
        """Write the object to ``fname`` (``.aa.ddm`` appended if missing) in the
        reference's file format (``azimuthalaverage.py:197-212``)."""
        from ._io import save_aa

        save_aa(self, fname)

    @property
    def shape(self) -> Tuple[int, int]:
        return self.data.shape


@dataclass
class BinSetup:
    """Host-side result of the binning set-up (``azimuthalaverage.py:349-432``)."""

    bin_edges: np.ndarray
    n_bins: int
    valid: np.ndarray      # flattened bool, pixel takes part
    bin_idx: np.ndarray    # flattened searchsorted index
    wi: np.ndarray         # flattened counts x weights
    sum_wi: np.ndarray
    sum_wi2: Optional[np.ndarray]
    k: np.ndarray


@dataclass
class BinArguments:
    """Checked arguments of the binning: edges, lower bound, mask and weights per pixel."""

    bin_edges: np.ndarray
    n_bins: int
    x_min: float
    mask: Optional[np.ndarray]   # bool, dist.shape; None: all pixels
    wi: np.ndarray               # counts x weights
    wi2: Optional[np.ndarray]    # counts x weights^2 (wi itself without weights), None without errors


def bin_arguments(dist: np.ndarray, bins, range, mask, weights, counts, eval_err: bool) -> BinArguments:
    """Validate the arguments; edges and weights per pixel."""
    m = None
    if mask is not None:
        m = mask.copy()
        if mask.shape != dist.shape:
            raise ValueError("mask shape and dist shape must be the same.")
        if mask.dtype != bool:
            m = mask.astype(bool)
            warnings.warn("mask is not of boolean type, it is cast to bool.")
    if weights is not None:
        if weights.shape != dist.shape:
            raise ValueError("weights shape and dist shape must be the same.")
        if np.any(weights < 0):
            raise ValueError("weights must be non-negative.")
    if counts is not None:
        if counts.shape != dist.shape:
            raise ValueError("counts shape and dist shape must be the same.")
    else:
        counts = np.ones(dist.shape, dtype=DTYPE)

    if range is None:
        x_min, x_max = np.min(dist), np.max(dist)
    else:
        x_min, x_max = range
        if x_min > x_max:
            x_min, x_max = x_max, x_min

    if isinstance(bins, int):
        edges = np.linspace(x_min, x_max, bins, dtype=DTYPE)
        n_bins = bins
    elif isinstance(bins, Iterable):
        # the same (for lists: lexicographic) comparison the reference applies
        if not np.all(bins[1:] >= bins[:-1]):
            raise ValueError("bins must be monotonically increasing.")
        edges = np.array(bins).astype(DTYPE)
        n_bins = len(bins)
        x_min = bins[0]
    else:
        raise ValueError("bins must be an int or an iterable.")

    wi = counts.astype(DTYPE)
    if weights is not None:
        wi *= weights
    wi2 = None
    if eval_err:
        wi2 = wi
        if weights is not None:
            wi2 = counts.astype(DTYPE)
            wi2 *= weights ** 2
    return BinArguments(edges, n_bins, x_min, m, wi, wi2)


def bin_setup(dist: np.ndarray, bins, range, mask, weights, counts, eval_err: bool) -> BinSetup:
    """Validate the arguments and compute edges, indices, weights and per-bin sums."""
    return bin_sums(dist, bin_arguments(dist, bins, range, mask, weights, counts, eval_err))


def bin_sums(dist: np.ndarray, args: BinArguments) -> BinSetup:
    """Bin indices and per-bin sums on the host."""
    edges, n_bins, wi, wi2 = args.bin_edges, args.n_bins, args.wi, args.wi2
    m = np.full(dist.shape, True) if args.mask is None else args.mask
    bin_idx = np.searchsorted(edges, dist)
    m[(bin_idx == n_bins) | (dist < args.x_min)] = False
    m[np.logical_not(wi)] = False

    valid = m.ravel()
    bidx = bin_idx.ravel()
    sel = bidx[valid]
    sum_wi = np.bincount(sel, weights=wi.ravel()[valid], minlength=n_bins).astype(DTYPE)[:n_bins]
    sum_wi2 = None
    if wi2 is not None:
        sum_wi2 = np.bincount(sel, weights=wi2.ravel()[valid], minlength=n_bins).astype(DTYPE)[:n_bins]
    with np.errstate(divide="ignore", invalid="ignore"):
        terms = dist.ravel()[valid] * wi.ravel()[valid] / sum_wi[sel]
    k = np.bincount(sel, weights=terms, minlength=n_bins).astype(DTYPE)[:n_bins]
    _fill_empty(k, sum_wi, edges)
    return BinSetup(edges, n_bins, valid, bidx, wi.ravel(), sum_wi, sum_wi2, k)


def _fill_empty(k: np.ndarray, sum_wi: np.ndarray, edges: np.ndarray) -> None:
    for b in np.flatnonzero(sum_wi == 0):
        k[b] = 0.5 * (edges[b - 1] + edges[b]) if b > 0 else edges[0]


# From this number of pixels on the device searches and sorts.  Set-up with uploads, host / device:
# 2112 pixels 0.28 / 0.28 ms, 4704 pixels 0.34 / 0.29, 131,584 pixels 4.4 / 0.59, 525,312 pixels 19.0 / 1.4.
DEVICE_BINS_PIXELS = 4096


def _longest_list(dist: np.ndarray, args: BinArguments) -> float:
    """The largest bin's share of the pixels, from a sample of 128."""
    at = np.arange(128) * 2654435761 % dist.size
    x = dist.take(at)
    inside = x >= args.x_min
    if args.mask is not None:
        inside &= args.mask.take(at)
    return np.bincount(np.searchsorted(args.bin_edges, x[inside]), minlength=args.n_bins + 1)[:args.n_bins].max() / 128.0


def _device_bins_faster(dist: np.ndarray, args: BinArguments) -> bool:
    """A bin's sums are chains of additions in pixel order, 60 ns a pixel and chain on the device (sum of w; of w2
    where it differs; of dist w / sum_w): with most pixels in one bin they outlast the host's whole set-up, 32 ns
    a pixel.  With s the largest bin's share and c chains, device and host were level at c s = 0.49 with 8320
    pixels, 0.56 with 33,024 and 0.64 with 525,312; the line lies 0.1 to 0.17 below, for the sample's error.
    525,312 pixels, set-up and the fast average, device / host: s = 1 65 / 23.6 ms, 0.6 40.5 / 23.0, 0.22 16.1 /
    22.9, 0.11 9.5 / 22.5; three chains, s = 0.22: 22.3 / 23.3."""
    chains = 2 if args.wi2 is None or args.wi2 is args.wi else 3
    return chains * _longest_list(dist, args) <= 0.5 - 1500.0 / dist.size


def _device_bins_usable(dist: np.ndarray, args: BinArguments) -> bool:
    """Whether fddm_b200_azimuthal_bins gives bin_sums' result (plain arrays, FP64 distances and bound, edges
    that are finite and in order: a list of edges may pass the argument check out of order), and sooner."""
    edges = args.bin_edges
    return (DEVICE_BINS_PIXELS <= dist.size < 2 ** 31 - 1024 and dist.dtype == np.float64
            and all(a is None or type(a) is np.ndarray for a in (dist, args.mask, args.wi, args.wi2, edges))
            and edges.ndim == 1 and 1 <= args.n_bins <= 16384 and len(edges) == args.n_bins
            and bool(np.all(np.isfinite(edges))) and bool(np.all(edges[1:] >= edges[:-1]))
            and isinstance(args.x_min, (int, float, np.integer, np.floating)) and bool(float(args.x_min) == args.x_min)
            and bool(_device_bins_faster(dist, args)))


@dataclass
class DeviceBins:
    """The tables of the average in device memory."""

    offsets: "torch.Tensor"
    pixels: "torch.Tensor"
    wi: "torch.Tensor"
    sum_wi: "torch.Tensor"
    bias: Optional["torch.Tensor"]
    mean: Optional["torch.Tensor"] = None  # sum dist w / sum_w where the device binned


def _upload(a: np.ndarray, device):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a if a.flags.writeable else a.copy()).to(device)


def _bins_on_device(dist: np.ndarray, args: BinArguments, device) -> DeviceBins:
    """bin_sums on the device (same bits: every sum adds in pixel order)."""
    npix, n_bins = dist.size, args.n_bins
    lib = _lib.load()
    need = ctypes.c_size_t()
    _lib.check(lib.fddm_b200_azimuthal_bins_workspace(npix, n_bins, ctypes.byref(need)))
    d_dist, d_w, d_edges = _upload(dist, device), _upload(args.wi, device).reshape(-1), _upload(args.bin_edges, device)
    d_w2 = None if args.wi2 is None or args.wi2 is args.wi else _upload(args.wi2, device)
    d_mask = None if args.mask is None else _upload(args.mask, device)
    scratch = torch.empty(need.value, dtype=torch.uint8, device=device)
    ints = torch.empty(n_bins + 1 + npix, dtype=torch.int32, device=device)
    sums = torch.empty((3, n_bins), dtype=torch.float64, device=device)
    res = DeviceBins(ints[:n_bins + 1], ints[n_bins + 1:], d_w, sums[0], None if args.wi2 is None else sums[1], sums[2])
    with torch.cuda.device(device):
        code = lib.fddm_b200_azimuthal_bins(
            d_dist.data_ptr(), d_w.data_ptr(), d_w2.data_ptr() if d_w2 is not None else None,
            d_mask.data_ptr() if d_mask is not None else None, npix, d_edges.data_ptr(), n_bins, float(args.x_min),
            scratch.data_ptr(), need.value, res.offsets.data_ptr(), res.pixels.data_ptr(), res.sum_wi.data_ptr(),
            res.bias.data_ptr() if res.bias is not None else None, res.mean.data_ptr(),
            torch.cuda.current_stream(device).cuda_stream,
        )
    _lib.check(code)
    return res


def _device_of(gpu_id):
    if torch is None or not torch.cuda.is_available():
        raise RuntimeError("the b200 azimuthal average needs a CUDA device (GB300)")
    return torch.device("cuda", int(gpu_id))


def _upload_bins(setup: BinSetup, eval_err: bool, device) -> DeviceBins:
    """Lists of the bins' pixels from the host's indices, and the tables in device memory."""
    n_bins = setup.n_bins
    pix = np.flatnonzero(setup.valid).astype(np.int32)
    key = setup.bin_idx[pix]
    # numpy sorts 16-bit keys by radix: 1.0 ms for 525,312 pixels where 64-bit ones took 5.5
    order = np.argsort(key.astype(np.uint16) if n_bins <= 0xFFFF else key, kind="stable")
    pix_sorted = pix[order]
    cnt = np.bincount(key, minlength=n_bins)[:n_bins]
    offsets = np.zeros(n_bins + 1, dtype=np.int32)
    np.cumsum(cnt, out=offsets[1:])
    bias = None
    if eval_err:
        with np.errstate(divide="ignore", invalid="ignore"):
            bias = np.where(setup.sum_wi > 0, setup.sum_wi - setup.sum_wi2 / setup.sum_wi, 0.0).astype(DTYPE)
    return DeviceBins(_upload(offsets, device), _upload(pix_sorted if len(pix_sorted) else np.zeros(1, np.int32), device),
                      _upload(setup.wi, device), _upload(setup.sum_wi, device),
                      _upload(bias, device) if eval_err else None)


def _bin_tables(dist: np.ndarray, args: BinArguments, eval_err: bool, device):
    """The average's tables on the device, and the host's set-up where that made them: the device's takes about 25
    bytes a pixel more while it runs, and where they are not there the host's still fits."""
    if _device_bins_usable(dist, args):
        try:
            return _bins_on_device(dist, args, device), None
        except torch.OutOfMemoryError:
            pass
    setup = bin_sums(dist, args)
    return _upload_bins(setup, eval_err, device), setup


def _average(data_dev, tables: DeviceBins, n_bins: int, eval_err: bool, device, exact: bool, host: bool):
    nrows = int(data_dev.shape[0])
    npix = int(np.prod(data_dev.shape[1:]))
    avg = torch.empty((n_bins, nrows), dtype=torch.float64, device=device)
    err = torch.empty((n_bins, nrows), dtype=torch.float64, device=device) if eval_err else None
    lib = _lib.load()
    data_dev = data_dev.contiguous()
    fn = lib.fddm_b200_azimuthal_average if exact else lib.fddm_b200_azimuthal_average_fast
    with torch.cuda.device(device):
        code = fn(
            data_dev.data_ptr(), nrows, npix, tables.offsets.data_ptr(), tables.pixels.data_ptr(), n_bins,
            tables.wi.data_ptr(), tables.sum_wi.data_ptr(), tables.bias.data_ptr() if tables.bias is not None else None,
            avg.data_ptr(), err.data_ptr() if err is not None else None, torch.cuda.current_stream(device).cuda_stream,
        )
    _lib.check(code)
    if not host:
        return avg, err
    return avg.cpu().numpy(), (err.cpu().numpy() if err is not None else None)


def azimuthal_average_array(
    data,
    dist: np.ndarray,
    bins: Optional[Union[int, Iterable[float]]] = 10,
    range: Optional[Tuple[float, float]] = None,
    mask: Optional[np.ndarray] = None,
    weights: Optional[np.ndarray] = None,
    counts: Optional[np.ndarray] = None,
    eval_err: Optional[bool] = True,
    *,
    gpu_id: int = 0,
    exact: bool = True,
) -> Tuple[np.ndarray, ...]:
    """Weighted azimuthal average of a 3D array (numpy, or a CUDA tensor already on the device).

    Returns ``(avg, err, k, bin_edges)``; ``avg``/``err`` have shape
    ``(n_bins, len(data))``, empty bins are NaN, ``err`` is None when
    ``eval_err`` is False.  ``exact=True`` reproduces the reference's per-pixel
    loops bit for bit; ``exact=False`` sums each bin with a warp of fused
    multiply-adds (rounding-level differences, much faster on large maps).
    """
    dim_y, dim_x = tuple(data.shape[-2:])
    if dist.shape != (dim_y, dim_x):
        raise ValueError("dist shape must be compatible with data shape.")
    eval_err = bool(eval_err)
    args = bin_arguments(dist, bins, range, mask, weights, counts, eval_err)
    device = _device_of(gpu_id)
    tables, setup = _bin_tables(dist, args, eval_err, device)
    if torch is not None and isinstance(data, torch.Tensor):
        data_dev = data.to(device=device, dtype=torch.float64)
    else:
        data_dev = torch.from_numpy(np.ascontiguousarray(data, dtype=np.float64)).to(device)
    avg, err = _average(data_dev, tables, args.n_bins, eval_err, device, exact, True)
    if setup is not None:
        return avg, err, setup.k, args.bin_edges
    k = tables.mean.cpu().numpy()
    _fill_empty(k, tables.sum_wi.cpu().numpy(), args.bin_edges)
    return avg, err, k, args.bin_edges


def azimuthal_average(
    img_str_func: ImageStructureFunction,
    bins: Optional[Union[int, Iterable[float]]] = 10,
    range: Optional[Tuple[float, float]] = None,
    mask: Optional[np.ndarray] = None,
    weights: Optional[np.ndarray] = None,
    eval_err: Optional[bool] = True,
    *,
    gpu_id: int = 0,
    exact: bool = True,
) -> AzimuthalAverage:
    """Azimuthal average of an image structure function (reference ``:481-564``).

    ``exact`` as in :func:`azimuthal_average_array`.

    Column 0 counts once, the last column once when the full width is even,
    every other column twice (its mirror image in the full plane).
    """
    counts = np.full(img_str_func.shape[1:], 2)
    counts[:, 0] = 1
    counts[:, -1] = 1 if img_str_func.width % 2 == 0 else 2
    gx, gy = np.meshgrid(img_str_func.kx, img_str_func.ky)
    k_modulus = np.sqrt(gx ** 2 + gy ** 2)
    data = img_str_func._device_data if img_str_func._device_data is not None else img_str_func._data
    avg, err, k, edges = azimuthal_average_array(
        data, k_modulus, bins, range, mask, weights, counts, eval_err, gpu_id=gpu_id, exact=exact
    )
    return AzimuthalAverage(avg, err, k, img_str_func.tau, edges)
