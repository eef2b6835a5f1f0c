"""Binning of craters that cover many bins: a layer of them has the heights that its windows have,
and takes the same time however its records lie side by side."""

import ctypes as C

import numpy as np
import pytest

from terraingen_b200 import _native as N
from terraingen_b200 import workloads as W
from terraingen_b200.device import centered

pytestmark = pytest.mark.gpu


def _apply(device, batch, grid, out):
    kernel, records, data, footprints = batch
    N.check(device._lib.tg_craters_apply(
        device._handle, kernel.ctypes.data, kernel.nbytes, records.ctypes.data, len(records),
        data.ctypes.data, len(data), footprints.ctypes.data, C.byref(grid), out.ctypes.data,
        N.NoData(0, 0.0), N.TG_MEMORY_HOST, None))


def _window(grid, col, row, side):
    return N.Grid(side, side, grid.origin_x + col * grid.pixel_width, grid.pixel_width, 0.0,
                  grid.origin_y + row * grid.pixel_height, 0.0, grid.pixel_height)


@pytest.mark.parametrize("general", [False, True], ids=["lean", "general"])
@pytest.mark.parametrize("smallest", [300.0, 40.0])
def test_a_layer_of_wide_craters_is_its_windows(device, smallest, general):
    spec = centered(1600, 1600, 1.0)
    batch = W.crater_batch(W.crater_population(5, 1.7, smallest, 500.0), spec,
                           shaping=W.config2_shaping())
    batch[0]["mantling"] = 1e-30 if general else 0.0
    grid = spec.native()
    whole = np.zeros((1600, 1600), np.float32)
    _apply(device, batch, grid, whole)
    assert np.abs(whole).max() > 1.0
    for col, row in ((0, 0), (768, 640), (1344, 1344)):  # 8 x 8 bins: none covers more
        part = np.zeros((256, 256), np.float32)
        _apply(device, batch, _window(grid, col, row, 256), part)
        np.testing.assert_array_equal(part, whole[row:row + 256, col:col + 256])


@pytest.mark.parametrize("general", [False, True], ids=["lean", "general"])
def test_craters_of_more_bins_than_a_block_takes_are_their_windows(device, general):
    """A grid of 9216 bins under craters that reach over all of it, among others."""
    spec = centered(3072, 3072, 0.5)
    batch = W.crater_batch(W.crater_population(5, 20.0, 100.0, 4000.0), spec)
    foot = batch[3].reshape(-1, 3)
    covering = np.abs(foot[:, :2]).max(axis=1) + 768.0 < foot[:, 2]
    assert 1 <= covering.sum() < len(foot)
    batch[0]["mantling"] = 1e-30 if general else 0.0
    grid = spec.native()
    whole = np.zeros((3072, 3072), np.float32)
    _apply(device, batch, grid, whole)
    assert np.abs(whole).max() > 1.0
    for col, row in ((0, 0), (1504, 2016), (2816, 2816)):
        part = np.zeros((256, 256), np.float32)
        _apply(device, batch, _window(grid, col, row, 256), part)
        np.testing.assert_array_equal(part, whole[row:row + 256, col:col + 256])


def _milliseconds(device, batch, spec):
    import torch

    kernel, records, data, footprints = batch
    inputs = (torch.from_numpy(records.view(np.uint8).copy()).cuda(),
              torch.from_numpy(data).cuda(), torch.from_numpy(footprints).cuda())
    heights = torch.zeros((spec.height, spec.width), device="cuda")
    best = np.inf
    for _ in range(12):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        device.craters_apply(kernel, *inputs[:2], spec, heights, footprints=inputs[2])
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_wide_craters_side_by_side_take_no_longer_than_apart(device):
    """128 craters of a meter whose footprints cover all 4096 bins of a grid: binning them is most
    of the call. Among 127 times as many records that lie off the grid it must not be faster."""
    spec = centered(2048, 2048, 1.0)
    kernel, records, data, footprints = W.crater_batch(
        W.crater_population(5, 0.02, 1.0, 4.0), spec, shaping=W.config2_shaping())
    foot = footprints.reshape(-1, 3)
    n = 128
    wide, around = foot[:n].copy(), np.array([0.0, 0.0, 4000.0])
    wide[:] = around
    apart_records = np.repeat(records[:n], 128)
    apart = np.tile(np.array([1e6, 1e6, 1.0]), (n * 128, 1))
    apart[::128] = around
    together = _milliseconds(device, (kernel, records[:n].copy(), data, wide.reshape(-1)), spec)
    spread = _milliseconds(device, (kernel, apart_records, data, apart.reshape(-1)), spec)
    print(f"side by side {together:.3f} ms, apart {spread:.3f} ms")
    assert together < 1.5 * spread
