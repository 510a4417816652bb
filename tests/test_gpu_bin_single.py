"""The smallest list that is not empty: one entry, in images whose tiles take no, one or two sorting passes."""
from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from realflare_gb300._abi import RasterArgs, check, lib  # noqa: E402
from realflare_gb300.device import empty, ptr, stream_handle  # noqa: E402


@pytest.mark.parametrize('size,tiles', [(16, 1), (32, 4), (64, 16), (256, 256), (272, 289)])
def test_one_entry(size, tiles):
    a = RasterArgs()
    a.width = a.height = size
    a.bin_size, a.tile_size = 32, 16
    a.path_count = a.wavelength_count = a.wavelength_sub_count = a.sub_steps = 1
    a.grid_count, a.screen_transform, a.ghost_width, a.ghost_height = 2, 1.0, 1, 1
    # a quad in the middle of the last tile, more than the bounds' 2 pixels inside it
    lo, hi = size - 12.0, size - 5.0
    vtx = torch.zeros((5, 8), device='cuda')
    # (the fifth vertex stands behind the last one, whose pair with one wavelength it ends)
    vtx[:, 0] = torch.tensor([lo, hi, lo, hi, hi])
    vtx[:, 1] = torch.tensor([lo, lo, hi, hi, hi])
    vtx[:4, 5] = 0.1
    bounds = torch.tensor([lo, lo, hi, hi], device='cuda') - size / 2
    nbytes, count = ctypes.c_size_t(), ctypes.c_int64()
    check(lib().rf_bin_workspace_size(ctypes.byref(a), 8, ctypes.byref(nbytes)), 'rf_bin_workspace_size')
    ws, offsets = empty((nbytes.value // 4 + 1,)), empty((tiles + 1,), torch.int32)
    entries = torch.full((8,), 77, dtype=torch.int32, device='cuda')  # (pair 0 is the only one there is)
    check(lib().rf_bin_tiles(ptr(bounds), ptr(vtx), ctypes.byref(a), ptr(ws), nbytes.value, ptr(offsets), ptr(entries),
                             8, ctypes.byref(count), stream_handle()), 'rf_bin_tiles')
    assert count.value == 1
    assert entries[0] == 0 and (entries[1:] == 77).all()
    assert offsets.tolist() == [0] * tiles + [1]
