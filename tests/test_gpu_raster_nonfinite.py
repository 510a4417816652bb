"""Records next to a vertex whose rrel or intensity is infinite (an element of height 0, a ray area of 0): mixed
over the wavelengths it is NaN, and the clamps of the falloff, the intensity and the reflectance make every
fragment 0. k_raster, which leaves the clamps out where no corner needs them, against rf_raster_masks,
which never does; the bound is the raster's in every other comparison."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import ghost_texture, rel_l2  # noqa: E402
from test_gpu_raster_quads import STAGE_RTOL, sheet  # noqa: E402

from realflare_gb300 import prepare  # noqa: E402
from realflare_gb300._abi import check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402

RREL, REFLECTANCE, INTENSITY = 4, 5, 6


@pytest.mark.parametrize('tile', [32, 16])
@pytest.mark.parametrize('field,value', [(RREL, np.inf), (INTENSITY, np.inf), (INTENSITY, np.nan), (INTENSITY, -1.0),
                                         (REFLECTANCE, np.inf)])
@pytest.mark.parametrize('wavelengths', [1, 3])
def test_clamps_act(wavelengths, field, value, tile):
    from oracle.oracle import Oracle
    from realflare_gb300.tasks import RasterizingTask

    o = Oracle('f32')
    rng = np.random.default_rng(11)
    p, rays = sheet(9, False, False, wavelengths, rng)
    rays[4] = rng.uniform(0.2, 0.9, rays[4].shape)  # every vertex well inside the housing
    G = p.render.grid_count
    area, min_area = prepare.quad_constants(p)
    bounds, inten = o.quad_setup(rays, 2, wavelengths, G, area, min_area)
    ghost, spec = ghost_texture(), light_spectrum()
    ra = prepare.raster_args(p, 2, wavelengths, ghost.shape, tile_size=tile)
    vtx = o.vertex(rays, inten, 2, wavelengths, G, ra.screen_transform, ra.width, ra.height)
    masks = o.bin_masks(bounds, ra.screen_transform, ra.width, ra.height, ra.bin_size)
    v = vtx.reshape(-1)[: 2 * G * G * wavelengths * 8].reshape(2, G * G, wavelengths, 8)
    v[:, rng.random(G * G) < 0.1, :, field] = value  # at all wavelengths

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    vtx_d, ghost_d, spec_d, masks_d = dev(vtx), dev(ghost), dev(spec), dev(masks.view(np.int64))
    offsets, entries = RasterizingTask().bin(ra, dev(bounds), vtx_d)
    image = torch.empty((ra.height, ra.width, 4), device='cuda')
    want = torch.empty_like(image)
    stream = int(torch.cuda.current_stream().cuda_stream)
    check(lib().rf_raster(vtx_d.data_ptr(), offsets.data_ptr(), entries.data_ptr(), ghost_d.data_ptr(),
                          spec_d.data_ptr(), ctypes.byref(ra), image.data_ptr(), stream), 'rf_raster')
    check(lib().rf_raster_masks(vtx_d.data_ptr(), masks_d.data_ptr(), masks.shape[1], ghost_d.data_ptr(),
                                spec_d.data_ptr(), ctypes.byref(ra), want.data_ptr(), stream), 'rf_raster_masks')
    got, want = image.cpu().numpy(), want.cpu().numpy()
    assert (want[..., :3] > 0).any()
    assert np.isfinite(got).all() and np.isfinite(want).all()
    assert rel_l2(got, want) < STAGE_RTOL
