"""Four samples per pixel on the made-up quads of test_gpu_raster_quads: their edge values are stepped from sample to
sample, a path of its own."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

import test_gpu_raster_quads as quads  # noqa: E402


@pytest.mark.parametrize('tile', [32, 16])
@pytest.mark.parametrize('wavelengths', [1, 2])
@pytest.mark.parametrize('clockwise', [False, True])
@pytest.mark.parametrize('cell,whole', [(2, True), (7, True), (8, False), (33, True), (40, False), (3000, False),
                                        (20000, False)])
def test_four_samples_match_oracle(cell, whole, clockwise, wavelengths, tile):
    quads.test_quads_match_oracle(cell, whole, clockwise, 4, wavelengths, tile)
