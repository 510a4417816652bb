"""The raster tile the library picks when the arguments leave it open (a host call, no GPU): 16
pixels where an image has too few 32-pixel tiles, 32 elsewhere, never a tile that does not divide
the bin, and never other than an explicit one."""
from __future__ import annotations

import ctypes
import os

import pytest

from realflare_gb300._abi import RasterArgs, RF_OK


def tile(width, height, samples=1, bin_size=64, explicit=0):
    from realflare_gb300 import build

    if not os.path.exists(build.LIB):
        build.build()
    lib = ctypes.CDLL(build.LIB)
    a = RasterArgs()
    a.width, a.height, a.bin_size, a.tile_size = width, height, bin_size, explicit
    a.path_count = a.wavelength_count = a.wavelength_sub_count = 1
    a.grid_count, a.sub_steps = 8, samples
    size, count = ctypes.c_int32(), ctypes.c_int32()
    status = lib.rf_raster_tiles(ctypes.byref(a), ctypes.byref(size), ctypes.byref(count))
    return size.value if status == RF_OK else None


@pytest.mark.parametrize('args,want', [
    ((7, 5), 16), ((640, 1024), 16), ((641, 1024), 32), ((1024, 1024), 32), ((2048, 2048), 32),
    ((1024, 1216, 2), 16), ((1025, 1216, 2), 32), ((1920, 1080, 4), 32),
    ((512, 512, 1, 32), 16), ((512, 512, 1, 16), None), ((512, 512, 1, 48), None), ((2048, 2048, 1, 48), None),
    ((512, 512, 1, 64, 32), 32), ((2048, 2048, 1, 64, 16), 16), ((512, 512, 1, 48, 16), 16),
])
def test_tile_rule(args, want):
    assert tile(*args) == want
