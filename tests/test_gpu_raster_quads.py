"""The rasteriser on made-up quads at the sizes and orientations where its branches meet.

A sheet of quads of a given cell size covers the image and its surroundings, counter-clockwise
or clockwise, with corners on whole pixels (samples fall on edges and vertices: the mean-value
weights' special cases) or not, rrel running through the housing's edge (0.9 to 1.05: records
inside, across and outside it), and with cells so large that coordinates leave the range where
edge functions are exact. The GPU image is compared with the oracle's, which shades every record
with the reference's arithmetic; the bound is the raster's in every other comparison (a few ulps
from the reciprocal and square-root instructions, summed over a pixel's fragments).
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import ghost_texture, reduced, rel_l2  # noqa: E402

from realflare_gb300 import prepare  # noqa: E402
from realflare_gb300._abi import check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402

STAGE_RTOL = 1e-5
SIZE = (101, 77)  # ragged against 16- and 32-pixel tiles and 8-pixel blocks


def sheet(cell: float, clockwise: bool, whole: bool, wavelengths: int, rng) -> tuple:
    """Six ray planes (pos, pos_apt, rrel, reflectance) of two sheets of quads, in mm."""
    w = reduced('plain-8', grid=3, resolution=SIZE, paths=2)
    p = w.project
    p.render.wavelengths = tuple(float(v) for v in np.linspace(420, 680, wavelengths))
    p.render.wavelength_count = wavelengths
    G = int(np.ceil(max(SIZE) / cell)) + 3
    p.render.grid_count = max(G, 4)
    G = p.render.grid_count
    st = prepare.raster_args(p, 2, wavelengths, (64, 64)).screen_transform
    iy, ix = np.mgrid[0:G, 0:G].astype(np.float64)
    rays = np.zeros((6, 2, wavelengths, G, G), np.float32)
    for k in range(2):
        for j in range(wavelengths):
            x = (ix - 1) * cell + 3 * j + 5 * k
            y = (iy - 1) * cell * (-1 if clockwise else 1) + (SIZE[1] if clockwise else 0) + 2 * j
            x, y = x + 0.25 * y * k, y + 0.125 * x * k  # the second sheet is sheared
            if not whole:
                x, y = x + rng.uniform(-0.3, 0.3, x.shape) * cell, y + rng.uniform(-0.3, 0.3, x.shape) * cell
            rays[0, k, j] = (np.round(x) if whole else x) / st - SIZE[0] / 2 / st
            rays[1, k, j] = (np.round(y) if whole else y) / st - SIZE[1] / 2 / st
    rays[2] = np.linspace(-0.9, 0.9, G)[None, None, None, :]
    rays[3] = np.linspace(-0.9, 0.9, G)[None, None, :, None]
    rays[4] = rng.uniform(0.9, 1.05, rays[4].shape)
    rays[4, :, :, : G // 2] = rng.uniform(0.2, 0.9, rays[4, :, :, : G // 2].shape)
    rays[5] = rng.uniform(0.0, 0.1, rays[5].shape)
    return p, rays.reshape(6, -1)


@pytest.mark.parametrize('tile', [32, 16])
@pytest.mark.parametrize('aa,wavelengths', [(1, 1), (1, 3), (2, 2), (8, 2)])
@pytest.mark.parametrize('clockwise', [False, True])
@pytest.mark.parametrize('cell,whole', [(2, True), (7, True), (8, False), (33, True), (40, False), (3000, False),
                                        (20000, False)])
def test_quads_match_oracle(cell, whole, clockwise, aa, wavelengths, tile):
    from oracle.oracle import Oracle
    from realflare_gb300.tasks import RasterizingTask

    o = Oracle('f32')
    p, rays = sheet(cell, clockwise, whole, wavelengths, np.random.default_rng(5))
    p.render.anti_aliasing = aa
    G = p.render.grid_count
    area, min_area = prepare.quad_constants(p)
    bounds, inten = o.quad_setup(rays, 2, wavelengths, G, area, min_area)
    ghost, spec = ghost_texture(), light_spectrum()
    ra = prepare.raster_args(p, 2, wavelengths, ghost.shape, tile_size=tile)
    vtx = o.vertex(rays, inten, 2, wavelengths, G, ra.screen_transform, ra.width, ra.height)
    masks = o.bin_masks(bounds, ra.screen_transform, ra.width, ra.height, ra.bin_size)
    want = o.raster(vtx, masks, ghost, spec, ra)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    vtx_d, ghost_d, spec_d = dev(vtx), dev(ghost), dev(spec)
    offsets, entries = RasterizingTask().bin(ra, dev(bounds), vtx_d)
    image = torch.empty((ra.height, ra.width, 4), device='cuda')
    check(lib().rf_raster(vtx_d.data_ptr(), offsets.data_ptr(), entries.data_ptr(), ghost_d.data_ptr(),
                          spec_d.data_ptr(), ctypes.byref(ra), image.data_ptr(),
                          int(torch.cuda.current_stream().cuda_stream)), 'rf_raster')
    torch.cuda.synchronize()
    got = image.cpu().numpy()
    assert np.isfinite(got).all() and np.abs(want).sum() > 0
    assert rel_l2(got, want) < STAGE_RTOL
