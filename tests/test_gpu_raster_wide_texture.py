"""Ghost textures with sides around 2^22 texels, past which a texel coordinate has no fraction of 23 bits: one quad
over the image, its fragments bilinear lookups of random texels in [1, 2], so each lies in [1, 2] (up to the
rounding of the sums) and together they spread over it; and one texture past 2^31 texels."""
from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from realflare_gb300._abi import RasterArgs, check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402


@pytest.mark.parametrize('width,height', [((1 << 22) - 1, 3), (1 << 22, 3), ((1 << 23) + 3, 2), (3, (1 << 23) + 3),
                                          (46341, 46341)])
@pytest.mark.parametrize('samples', [1, 2])
def test_lookups_interpolate(width, height, samples):
    from realflare_gb300.tasks import RasterizingTask

    if torch.cuda.mem_get_info()[0] < 16 * width * height:
        pytest.skip('not enough device memory')
    a = RasterArgs()
    a.width = a.height = 64
    a.bin_size, a.tile_size, a.sub_steps = 64, 32, samples
    a.path_count = a.wavelength_count = a.wavelength_sub_count = 1
    a.grid_count, a.screen_transform, a.intensity, a.ghost_scale = 2, 1.0, 1.0, 1.0
    a.ghost_width, a.ghost_height = width, height
    vtx = torch.zeros((5, 8), device='cuda')
    vtx[:, 0] = torch.tensor([-9.0, 73.0, -9.0, 73.0, 73.0])
    vtx[:, 1] = torch.tensor([-9.0, -9.0, 73.0, 73.0, 73.0])
    across = width > height  # inside the texture along its long side, in the middle of the short one
    vtx[:, 2 if across else 3] = torch.tensor([-0.9, 0.9, -0.9, 0.9, 0.9])
    vtx[:, 4], vtx[:, 5], vtx[:, 6] = 0.5, 0.5, 2.0
    bounds = torch.tensor([-41.0, -41.0, 41.0, 41.0], device='cuda')
    ghost = 1 + torch.rand((height, width), device='cuda', generator=torch.Generator('cuda').manual_seed(4))
    spectrum = torch.from_numpy(light_spectrum()).cuda()
    offsets, entries = RasterizingTask().bin(a, bounds, vtx)
    image = torch.empty((64, 64, 4), device='cuda')
    flat = torch.ones((1, 1), device='cuda')  # one texel of 1: its lookups at the middle of the image give the scale
    stream = int(torch.cuda.current_stream().cuda_stream)
    check(lib().rf_raster(vtx.data_ptr(), offsets.data_ptr(), entries.data_ptr(), ghost.data_ptr(), spectrum.data_ptr(),
                          ctypes.byref(a), image.data_ptr(), stream), 'rf_raster')
    vtx[:, 2:4] = 0.0
    a.ghost_width = a.ghost_height = 1
    one = torch.empty_like(image)
    check(lib().rf_raster(vtx.data_ptr(), offsets.data_ptr(), entries.data_ptr(), flat.data_ptr(), spectrum.data_ptr(),
                          ctypes.byref(a), one.data_ptr(), stream), 'rf_raster')
    lookups = (image / one)[..., 0]
    assert lookups.min() > 1 - 1e-5 and lookups.max() < 2 + 1e-5
    assert lookups.max() - lookups.min() > 0.5
