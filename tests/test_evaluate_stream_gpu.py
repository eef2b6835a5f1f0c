"""tg_evaluate on device memory bins its layers on a stream of the device's own, beside the source on
the caller's: binning that has to grow its entries and run again, and inputs that the caller's
stream is still to write."""

import numpy as np
import pytest

from terraingen_b200 import workloads as W
from terraingen_b200.device import centered

pytestmark = pytest.mark.gpu


def _scene():
    """A layer of craters and boulders that cover most bins of a grid each."""
    grid = centered(1024, 1024, 1.0)
    craters = W.crater_batch(W.crater_population(5, 1.7, 200.0, 500.0), grid,
                             shaping=W.config2_shaping())
    stones = np.zeros((13, 5), np.float64)
    stones[:, 0] = np.linspace(-10.0, 10.0, 13)
    stones[:, 2] = 1500.0
    stones[:, 3:] = 1.0
    return grid, craters, stones, np.array([W.fractal(seed=7, wavelength=512.0, amplitude=5.0,
                                                      octaves=8)])


def _tensors(craters, stones):
    import torch

    _, records, data, footprints = craters
    return [torch.from_numpy(a.copy()).cuda()
            for a in (records.view(np.uint8), data, footprints, stones)]


def _evaluate(device, scene, tensors, heights):
    grid, craters, _, fractals = scene
    records, data, footprints, stones = tensors
    return device.evaluate(grid, heights, fractals=fractals,
                           craters=(craters[0], records, data, footprints), boulders=stones,
                           boulder_width=grid.pixel)


def test_growing_on_device_memory_gives_the_same_heights():
    import torch

    from terraingen_b200 import Device

    scene = _scene()
    grid = scene[0]
    tensors = _tensors(*scene[1:3])
    with Device() as fresh:  # its entries' first capacity is a guess that this layer outgrows
        first, again = (torch.full((grid.height, grid.width), 7.0, device="cuda")
                        for _ in range(2))
        _evaluate(fresh, scene, tensors, first)
        pairs = fresh.counters()
        _evaluate(fresh, scene, tensors, again)
        assert fresh.counters() == pairs and pairs["crater_pairs"] > 0
    assert torch.equal(first.view(torch.int32), again.view(torch.int32))
    host = np.zeros((grid.height, grid.width), np.float32)
    with Device() as fresh:
        fresh.evaluate(grid, host, fractals=scene[3], craters=scene[1], boulders=scene[2],
                       boulder_width=grid.pixel)
    np.testing.assert_array_equal(first.cpu().numpy(), host)


def test_inputs_the_stream_is_still_to_write_are_waited_for(device):
    import torch

    scene = _scene()
    grid, _, _, _ = scene
    ready = _tensors(*scene[1:3])
    want = _evaluate(device, scene, ready, torch.empty((grid.height, grid.width), device="cuda"))
    # Other inputs of the same sizes, as valid: the craters and boulders without any relief.
    flat = _tensors(*scene[1:3])
    records, _, _, stones = flat
    records.view(-1, 144)[:] = records.view(-1, 144)[0].clone()
    flat[2].view(-1, 3)[:] = torch.tensor([1e6, 1e6, 1.0], dtype=torch.float64, device="cuda")
    stones[:, 0] = 1e6
    other = _evaluate(device, scene, flat, torch.empty_like(want))
    assert not torch.equal(other, want)
    got = torch.empty_like(want)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)  # 10 ms at 2 GHz, before the copies
        for to, of in zip(flat, ready):
            to.copy_(of)
        _evaluate(device, scene, flat, got)
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
