"""A frame's image is the same bit for bit in 16- and in 32-pixel tiles, single and batched: also where quads reach
4096 samples and more beyond the image, from where on the products of the mean-value weights round."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import ghost_texture  # noqa: E402
from test_gpu_raster_quads import sheet  # noqa: E402

from realflare_gb300 import prepare  # noqa: E402
from realflare_gb300._abi import check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402


@pytest.mark.parametrize('aa', [1, 2, 4, 8])
@pytest.mark.parametrize('cell', [7, 3000, 7000, 20000])
@pytest.mark.parametrize('clockwise', [False, True])
def test_tiles_give_the_same_bits(clockwise, cell, aa):
    from oracle.oracle import Oracle
    from realflare_gb300.tasks import RasterizingTask

    o = Oracle('f32')
    p, rays = sheet(cell, clockwise, False, 3, np.random.default_rng(8))
    p.render.anti_aliasing = aa
    G = p.render.grid_count
    area, min_area = prepare.quad_constants(p)
    bounds, inten = o.quad_setup(rays, 2, 3, G, area, min_area)
    ghost, spec = (torch.from_numpy(a).cuda() for a in (ghost_texture(), light_spectrum()))
    images = []
    for tile in (16, 32):
        ra = prepare.raster_args(p, 2, 3, tuple(ghost.shape), tile_size=tile)
        vtx = torch.from_numpy(o.vertex(rays, inten, 2, 3, G, ra.screen_transform, ra.width, ra.height)).cuda()
        offsets, entries = RasterizingTask().bin(ra, torch.from_numpy(bounds).cuda(), vtx)
        image = torch.empty((ra.height, ra.width, 4), device='cuda')
        check(lib().rf_raster(vtx.data_ptr(), offsets.data_ptr(), entries.data_ptr(), ghost.data_ptr(), spec.data_ptr(),
                              ctypes.byref(ra), image.data_ptr(), int(torch.cuda.current_stream().cuda_stream)),
              'rf_raster')
        images.append(image)
    assert images[0].abs().sum() > 0
    assert torch.equal(*images)


@pytest.mark.parametrize('samples', [(1, 1, 1, 1), (1, 4, 1, 2)])
def test_batch_of_a_small_frame_is_the_single_frame(samples):
    """16-pixel tiles alone, 32-pixel ones in the batch; a long lens throws its ghosts far beyond the image. Mixed
    samples take the batch kernel with the sample count at run time."""
    from realflare_gb300 import synthetic
    from realflare_gb300.batch import BatchRenderer, ghost_textures
    from realflare_gb300.device import Image
    from realflare_gb300.tasks import RasterizingTask, RaytracingTask

    projects = synthetic.batched_projects(4, seed=3, resolution=448, surfaces=(16, 24), grids=(8, 12))
    for p, aa in zip(projects, samples):
        p.render.anti_aliasing = aa
    tex, offs, shapes = ghost_textures(projects)
    images = BatchRenderer(projects, tile_size=32, rays_per_thread=2, ghosts=(tex, offs, shapes)).run()
    torch.cuda.synchronize()
    task = RasterizingTask()
    for p, img, off, (h, w) in zip(projects, images, offs, shapes):
        want = task.run(p, RaytracingTask(cache=False).run(p), Image(tensor=tex[off: off + h * w].view(h, w))).tensor
        assert task.tile_size == 16 and want.abs().sum() > 0
        assert torch.equal(img, want)
