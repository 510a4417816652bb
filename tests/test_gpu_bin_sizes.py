"""Binning where its launches change form: tile counts around one scan block, one order block and the widths of
the packed rectangles, pairs around a block of 256, against a plain evaluation of the lists."""

import ctypes

import numpy as np
import pytest
import torch

from realflare_gb300._abi import RasterArgs, check, lib
from realflare_gb300.device import empty, ptr, stream_handle

pytestmark = pytest.mark.gpu


def rectangles(bounds, vtx, a, tile):
    """Tile rectangles of every pair, in the reference's bins and the pair's pixel bounds widened by 2."""
    ntx, nty = -(-a.width // tile), -(-a.height // tile)
    bdx, bdy = -(-a.width // a.bin_size), -(-a.height // a.bin_size)
    g, per = a.grid_count, a.bin_size // tile
    quads = (g - 1) ** 2
    out = []
    for prim in range(a.path_count * quads):
        s = np.trunc(bounds[prim] * np.float32(a.screen_transform)).astype(np.int64)
        s += np.array([a.width // 2, a.height // 2] * 2)
        bx = max((s[0] - 1) // a.bin_size, 0), min(s[2] // a.bin_size, bdx - 1)
        by = max((s[1] - 1) // a.bin_size, 0), min(s[3] // a.bin_size, bdy - 1)
        path, quad = divmod(prim, quads)
        c0 = (quad // (g - 1)) * g + quad % (g - 1)
        for w in range(max(a.wavelength_count - 1, 1)):
            base = [(path * g * g + c) * a.wavelength_count + w for c in (c0, c0 + 1, c0 + 1 + g, c0 + g)]
            p = np.concatenate([vtx[[b, b + 1], :2] for b in base])
            lo = np.floor((p.min(0) - np.float32(2)) / np.float32(tile)).astype(int)
            hi = np.floor((p.max(0) + np.float32(2)) / np.float32(tile)).astype(int)
            tx = max(bx[0] * per, lo[0]), min((bx[1] + 1) * per - 1, ntx - 1, hi[0])
            ty = max(by[0] * per, lo[1]), min((by[1] + 1) * per - 1, nty - 1, hi[1])
            out.append((tx, ty) if bx[0] <= bx[1] and by[0] <= by[1] else ((0, -1), (0, -1)))
    return out, ntx, nty


@pytest.mark.parametrize('width, height, tile, bin_size, grid, paths, wavelengths', [
    (16, 16, 16, 32, 2, 1, 1),        # one tile, one pair
    (17, 2049, 16, 32, 2, 3, 2),      # two columns of tiles
    (4096, 16, 16, 32, 3, 64, 2),     # one row: 256 pairs, 256 tiles
    (2050, 2050, 16, 32, 4, 29, 2),   # 16641 tiles: more than one order block; 261 pairs
    (16000, 24, 32, 64, 5, 33, 3),    # wide and low
    (4096, 1030, 32, 32, 6, 21, 4),   # 4224 tiles: keys of 13 bits
])
def test_lists(width, height, tile, bin_size, grid, paths, wavelengths):
    a = RasterArgs()
    a.width, a.height, a.bin_size, a.tile_size = width, height, bin_size, tile
    a.sub_steps = a.wavelength_sub_count = 1
    a.path_count, a.grid_count, a.wavelength_count = paths, grid, wavelengths
    a.screen_transform = 1.0
    a.ghost_width = a.ghost_height = 1
    rng = np.random.default_rng(width + paths)
    n = paths * grid * grid * wavelengths + 1
    vtx = np.zeros((n, 8), np.float32)
    vtx[:, 0] = rng.uniform(-20, width + 20, n) if width < 4096 else np.clip(rng.normal(width / 2, width / 50, n), 0, width)
    vtx[:, 1] = rng.uniform(-20, height + 20, n) if height < 2050 else np.clip(rng.normal(height / 2, 40, n), 0, height)
    vtx[:, 5] = 0.1
    quads = (grid - 1) ** 2
    bounds = np.empty((paths * quads, 4), np.float32)
    for prim in range(len(bounds)):
        path, quad = divmod(prim, quads)
        c0 = (quad // (grid - 1)) * grid + quad % (grid - 1)
        rows = [(path * grid * grid + c) * wavelengths + w for c in (c0, c0 + 1, c0 + 1 + grid, c0 + grid)
                for w in range(wavelengths)]
        p = vtx[rows, :2] - np.array([width / 2, height / 2], np.float32)
        bounds[prim] = (*p.min(0), *p.max(0))
    bounds[rng.random(len(bounds)) < 0.2, 0] = np.nan
    b = np.where(np.isnan(bounds), np.float32(1e9), bounds)  # a culled primitive: beyond the image, no bins
    rects, ntx, nty = rectangles(b, vtx, a, tile)
    lists = [[] for _ in range(ntx * nty)]
    for pair, (tx, ty) in enumerate(rects):
        for y in range(ty[0], ty[1] + 1):
            for x in range(tx[0], tx[1] + 1):
                lists[y * ntx + x].append(pair)
    total = sum(map(len, lists))
    bd, vd = torch.from_numpy(bounds).cuda(), torch.from_numpy(vtx).cuda()
    size, count = ctypes.c_size_t(), ctypes.c_int64()
    check(lib().rf_bin_workspace_size(ctypes.byref(a), total, ctypes.byref(size)), 'rf_bin_workspace_size')
    ws = empty((size.value // 4 + 1,))
    offsets, entries = empty((ntx * nty + 1,), torch.int32), empty((max(total, 1),), torch.int32)
    check(lib().rf_bin_tiles(ptr(bd), ptr(vd), ctypes.byref(a), ptr(ws), size.value, ptr(offsets), ptr(entries), total,
                             ctypes.byref(count), stream_handle()), 'rf_bin_tiles')
    assert count.value == total > 0
    starts = np.concatenate([[0], np.cumsum([len(x) for x in lists])])
    assert np.array_equal(offsets.cpu().numpy(), starts)
    assert np.array_equal(entries[:total].cpu().numpy(), np.concatenate([np.array(x, int) for x in lists]))
    # the raster's order: decreasing counts within an eighth of a power of two, ties by tile
    tiles = ntx * nty
    check(lib().rf_tile_order_workspace_size(tiles, ctypes.byref(size)), 'rf_tile_order_workspace_size')
    ows, order = empty((size.value // 4 + 1,)), empty((tiles,), torch.int32)
    check(lib().rf_tile_order(ptr(offsets), tiles, ptr(ows), size.value, ptr(order), stream_handle()), 'rf_tile_order')
    def key(k):
        e = k.bit_length() - 1
        return 255 if k == 0 else 255 - (8 * e + ((k << 3 >> e) & 7))
    keys = np.array([key(len(x)) for x in lists])
    assert np.array_equal(order.cpu().numpy(), np.argsort(keys, kind='stable'))
