"""One RasterizingTask for images of different tile counts (a host call, no GPU): the order is made for the
tiles the image has, not for those of a larger list an earlier image left in the task's buffers."""
from __future__ import annotations

import ctypes
import os

import pytest

torch = pytest.importorskip('torch')

from realflare_gb300 import tasks  # noqa: E402
from realflare_gb300._abi import RF_OK, RasterArgs  # noqa: E402


class HostCalls:
    """The library's host calls, with its device calls recorded instead of run."""

    def __init__(self) -> None:
        from realflare_gb300 import build

        if not os.path.exists(build.LIB):
            build.build()
        lib = ctypes.CDLL(build.LIB)
        self.rf_raster_tiles, self.rf_bin_workspace_size = lib.rf_raster_tiles, lib.rf_bin_workspace_size
        self.rf_tile_order_workspace_size = lib.rf_tile_order_workspace_size
        self.rf_bin_workspace_size.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
        self.ordered = []

    def rf_bin_tiles(self, *args) -> int:
        return RF_OK

    def rf_tile_order(self, offsets, tiles, *args) -> int:
        self.ordered.append(tiles)
        return RF_OK


@pytest.mark.parametrize('sizes', [
    [(640, 640, 1), (1024, 1024, 1)],   # 1600 tiles of 16 pixels, then 1024 of 32
    [(1024, 1024, 4), (1024, 1024, 1)],  # the same image with other samples
    [(300, 200, 1), (40, 30, 1), (300, 200, 1)],
    [(2048, 2048, 1), (7, 5, 1)],
])
def test_order_covers_the_images_tiles(sizes, monkeypatch):
    monkeypatch.setattr(tasks, 'empty', lambda shape, dtype=torch.float32: torch.empty(shape, dtype=dtype))
    monkeypatch.setattr(tasks.Task, 'stream', property(lambda self: 0))
    monkeypatch.setattr(tasks.Task, '__init__', lambda self, queue=None: setattr(self, 'lib', HostCalls()))
    task = tasks.RasterizingTask()
    for width, height, samples in sizes:
        a = RasterArgs()
        a.width, a.height, a.bin_size, a.sub_steps = width, height, 64, samples
        a.path_count = a.wavelength_count = a.wavelength_sub_count = 1
        a.grid_count = 8
        count = ctypes.c_int32()
        assert task.lib.rf_raster_tiles(ctypes.byref(a), None, ctypes.byref(count)) == RF_OK
        offsets, _ = task.bin(a, None, None)
        assert offsets.numel() == count.value + 1
        task.order(offsets)
        assert task.lib.ordered[-1] == count.value
