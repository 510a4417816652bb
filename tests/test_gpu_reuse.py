"""One engine for several image sizes and sample counts: every image equals a fresh engine's bit for bit, also
where a later image has fewer raster tiles than an earlier one."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import reduced  # noqa: E402

from realflare_gb300.data import QSize, RenderElement  # noqa: E402


@pytest.mark.parametrize('settings', [
    [(640, 640, 1), (1024, 1024, 1), (640, 640, 1)],   # 1600 tiles, then 1024
    [(1024, 1024, 4), (1024, 1024, 1)],                # 4096, then 1024
    [(1500, 900, 1), (33, 47, 2), (400, 300, 1)],      # a large image, then small ones
])
def test_engine_reused(settings):
    from realflare_gb300.engine import Engine

    p = reduced('plain-8', grid=16).project
    p.output.element = RenderElement.FLARE

    def image(engine, width, height, samples):
        p.render.resolution = QSize(width, height)
        p.render.anti_aliasing = samples
        assert engine.render(p)
        return engine.image.tensor

    one = Engine()
    for s in settings:
        got, want = image(one, *s), image(Engine(), *s)
        assert want.abs().sum() > 0
        assert torch.equal(got, want)
