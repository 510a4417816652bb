"""rf_raster_backward into gradient buffers of every alignment a float buffer can have: the vector additions of
the aligned form and the scalar ones of the others give the same sums, in an unspecified order of additions
(a vertex sums some hundred terms: rounding 1e-5 of the whole at most). A buffer that is no float's is refused."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import ghost_texture, oracle_pipeline, reduced  # noqa: E402

from realflare_gb300._abi import RF_OK, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402

RF_ERR_INVALID_ARG = 1


@pytest.mark.parametrize('aa,tile', [(1, 32), (1, 16), (2, 16)])
def test_any_float_alignment(aa, tile):
    from oracle.oracle import Oracle
    from realflare_gb300.tasks import RasterizingTask

    w = reduced('spectral-16', grid=12, resolution=(100, 80), paths=12, wavelengths=3)
    w.project.render.anti_aliasing = aa
    w.project.render.wavelength_sub_count = 2
    ghost, spec = ghost_texture(), light_spectrum()
    r = oracle_pipeline(Oracle('f32'), w, ghost, spec)
    ra = r['raster_args']
    ra.tile_size = tile
    vtx, bounds, ghost, spec = (torch.from_numpy(np.ascontiguousarray(a)).cuda()
                                for a in (r['vtx'], r['bounds'], ghost, spec))
    offsets, entries = RasterizingTask().bin(ra, bounds, vtx)
    stream = int(torch.cuda.current_stream().cuda_stream)
    image = torch.empty((ra.height, ra.width, 4), device='cuda')
    lists = (vtx.data_ptr(), offsets.data_ptr(), entries.data_ptr(), ghost.data_ptr(), spec.data_ptr(), ctypes.byref(ra))
    assert lib().rf_raster(*lists, image.data_ptr(), stream) == RF_OK
    grad_image = torch.randn(image.shape, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    n = vtx.numel()

    def backward(offset):  # in floats
        buffer = torch.full((n + 8,), 5.0, device='cuda')
        status = lib().rf_raster_backward(*lists, image.data_ptr(), grad_image.data_ptr(),
                                          buffer.data_ptr() + int(4 * offset), stream)
        return status, buffer

    status, want = backward(0)
    assert status == RF_OK
    want = want[:n].double()
    assert want.abs().sum() > 0
    for offset in (1, 2, 3, 4):
        status, buffer = backward(offset)
        assert status == RF_OK
        assert (buffer[:offset] == 5).all() and (buffer[offset + n:] == 5).all()
        assert (buffer[offset:offset + n].double() - want).norm() <= 1e-5 * want.norm()
    status, buffer = backward(0.5)
    assert status == RF_ERR_INVALID_ARG and (buffer == 5).all()
