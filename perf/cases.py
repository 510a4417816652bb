"""The render path's timing cases: what is rendered, how a program calls it, and the same values in
64 bits where a plain evaluation of them is affordable.

Families (``kind``):

* ``render``: ``Engine.render`` of one project, the call every user makes. The element is a
  ghost texture (the smallest call: an aperture mask and its diffraction), a starburst, a flare
  (trace, quad setup, binning, raster) or both composited.
* ``raster``: ``RasterizingTask.run`` on traced rays and a ghost texture (a program that keeps its
  rays and changes raster settings).
* ``trace``: ``RaytracingTask.run``, FP32 or with double-precision ray geometry.
* ``batch``: a replay of ``BatchRenderer``'s captured frames (many lights and lenses at once).
* ``adjoint``: a training step of the differentiable flare: image, then the gradients of an image
  loss with respect to radii, gaps, coating thicknesses and light position.

The engine is made without its trace cache: a pass is what a changed project costs. Seeds move the
light, the ghost aperture and the dust; the lenses are the workloads' own.
"""
from __future__ import annotations

import copy
import math

import numpy as np
import torch

from realflare_gb300 import prepare as host
from realflare_gb300 import synthetic
from realflare_gb300.batch import BatchRenderer
from realflare_gb300.constants import light_spectrum
from realflare_gb300.data import (
    Aperture,
    ApertureDust,
    ApertureShape,
    FlareLens,
    Project,
    QPointF,
    QSize,
    QSizeF,
    RenderElement,
)
from realflare_gb300.device import Image
from realflare_gb300.diff import DifferentiableRenderer
from realflare_gb300.engine import Engine
from realflare_gb300.tasks import GhostApertureTask, GhostTask, RasterizingTask, RaytracingTask

DEVICE = 'cuda'
WORKLOADS = {8: 'plain-8', 16: 'spectral-16', 24: 'production-24'}
LIGHTS = {8: (0.2, 0.1), 16: (0.35, -0.2), 24: (0.3, 0.2), 50: (0.6, 0.3)}
GHOSTS = {8: 28, 16: 120, 24: 276, 50: 91}
ELEMENTS = {8: 10, 16: 18, 24: 26, 50: 30}
# coating wavelengths (nm) of the bundled 50-135 mm zoom in the reference's benchmark project
ZOOM_COATING = (544, 558, 460, 690, 488, 430, 526, 540, 676, 590, 539, 518, 561, 685, 462, 534, 639, 456, 422, 447,
                393, 522, 610, 475, 674, 596, 475, 488, 645, 526)
# a fragment's FP32 operations (mean-value weights 67, shading 71, colour 12) and a surface
# interaction's (intersection, refraction; the two reflections of a path spread over its steps)
FRAGMENT_FLOPS, INTERACTION_FLOPS = 150, 90


def listed() -> list:
    return [
        # one ghost texture at the default size: what an interactive host asks for most often
        dict(name='ghost-256', kind='render', element='GHOST', ghost_w=256, ghost_h=256),
        # the starburst of a small preview, with the jitter and rotation that soften its spikes
        dict(name='starburst-preview', kind='render', element='STARBURST', width=512, height=512, star_w=256,
             star_h=256, samples=100, blur=1.0, rotation=5.0),
        # one diffraction pattern per wavelength, full HD, dust on the aperture, no jitter
        dict(name='starburst-1080', kind='render', element='STARBURST', width=1920, height=1080, star_w=512,
             star_h=512, samples=100, dust=True, spectra=16),
        # the smallest flare workload: 8 surfaces, 28 ghosts, one wavelength
        dict(name='flare-8', kind='render', element='FLARE', lens=8, grid=32, wavelengths=1, width=512, height=512),
        # the mid-size flare workload: 16 surfaces, 120 ghosts, 8 wavelengths
        dict(name='flare-16', kind='render', element='FLARE', lens=16, grid=64, wavelengths=8, width=1024,
             height=1024),
        # the production frame: 24 surfaces, 276 ghosts, 16 wavelengths, two-layer coatings, starburst
        dict(name='frame-24', kind='render', element='FLARE_STARBURST', lens=24, grid=128, wavelengths=16,
             width=2048, height=2048, star_w=512, star_h=512, samples=100, dust=True),
        # the reference's own benchmark project: a zoom lens, half its ghosts culled, 4 samples per
        # pixel, 8 sub-steps per wavelength, 1000 jittered starburst samples
        dict(name='zoom-1080', kind='render', element='FLARE_STARBURST', lens=50, grid=129, wavelengths=5, sub=8,
             aa=4, width=1920, height=1080, ghost_w=512, ghost_h=512, star_w=512, star_h=512, samples=1000, blur=1.0),
        # a raster of odd sizes throughout, 2 samples per pixel and 2 sub-steps
        dict(name='raster-ragged', kind='raster', lens=8, grid=45, wavelengths=3, sub=2, aa=2, width=601, height=403,
             ghost_w=300, ghost_h=200),
        # a trace whose grid is no multiple of anything
        dict(name='trace-16', kind='trace', lens=16, grid=97, wavelengths=7),
        # the opt-in double-precision trace
        dict(name='trace-accurate', kind='trace', lens=16, grid=33, wavelengths=4, accurate=True),
        # an animation's or a light field's frames, rendered together
        dict(name='batch-12', kind='batch', frames=12, width=512, height=512, grid=64, wavelengths=8),
        # one step of fitting a lens to an image
        dict(name='adjoint-16', kind='adjoint', lens=16, grid=64, wavelengths=8, width=512, height=512),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """A case of the listed ones' ranges, no dearer than the production frame."""
    limit = _fragments(listed()[5]) / 2
    while True:
        kind = rng.choice(['ghost', 'starburst', 'flare', 'flare', 'flare', 'raster', 'trace', 'batch', 'adjoint'])
        size = dict(width=_log(rng, 128, 2048), height=_log(rng, 128, 2048))
        scene = dict(lens=rng.choice([8, 16, 24]), grid=_log(rng, 16, 128), wavelengths=_log(rng, 1, 16))
        ghost = dict(ghost_w=_log(rng, 64, 512), ghost_h=_log(rng, 64, 512))
        if kind == 'ghost':
            return dict(kind='render', element='GHOST', ghost_w=_log(rng, 64, 1024), ghost_h=_log(rng, 64, 1024))
        if kind == 'starburst':
            return dict(kind='render', element='STARBURST', **size, star_w=_log(rng, 64, 512),
                        star_h=_log(rng, 64, 512), samples=_log(rng, 50, 400), blur=rng.choice([0.0, 1.0]),
                        rotation=rng.choice([0.0, 0.0, 5.0]), dust=rng.random() < 0.5,
                        spectra=rng.choice([1, _log(rng, 2, 16)]))
        if kind == 'flare':
            case = dict(kind='render', element='FLARE', **scene, **size, **ghost, aa=rng.choice([1, 1, 2, 4]),
                        sub=rng.choice([1, 1, 2, 4]))
        elif kind == 'raster':
            case = dict(kind='raster', **scene, **size, **ghost, aa=rng.choice([1, 2, 4]), sub=rng.choice([1, 2]))
        elif kind == 'trace':
            accurate = rng.random() < 0.3
            case = dict(kind='trace', **scene, accurate=accurate)
            if accurate:
                case.update(grid=_log(rng, 16, 33), wavelengths=_log(rng, 1, 8))
            return case
        elif kind == 'batch':
            side = _log(rng, 128, 768)
            case = dict(kind='batch', frames=rng.randint(2, 16), width=side, height=side, grid=_log(rng, 16, 64),
                        wavelengths=_log(rng, 1, 8))
        else:
            case = dict(kind='adjoint', lens=rng.choice([8, 16]), grid=_log(rng, 16, 64),
                        wavelengths=_log(rng, 2, 8), width=_log(rng, 64, 512), height=_log(rng, 64, 512))
        if _fragments(case) * case.get('aa', 1) <= limit:
            return case


# ------------------------------------------------------------------------------ inputs
def _wavelengths(n: int) -> tuple:
    return (550.0,) if n == 1 else tuple(float(v) for v in np.linspace(390.0, 700.0, n))


def _lens(surfaces: int) -> FlareLens:
    if surfaces == 50:
        return FlareLens(sensor_size=QSizeF(36, 24), fstop=4.8, lens_model_path='$RES/model/Nikon/ai_50_135mm.json',
                         glasses_path='$RES/glass/schott', coating=ZOOM_COATING, min_area=0.1)
    return copy.deepcopy(synthetic.workload(WORKLOADS[surfaces]).project.flare.lens)


def _project(case: dict, seed: int) -> Project:
    """The project of a case: its sizes and options, and the seed's light, ghost iris and dust."""
    rng = np.random.Generator(np.random.PCG64(seed))
    move = rng.uniform(-0.05, 0.05, 2)
    rotation, fstop, dust_seed = float(rng.uniform(0, 45)), float(rng.uniform(2.0, 16.0)), int(rng.integers(1 << 30))
    surfaces = case.get('lens', 8)
    p = Project()
    p.output.element = RenderElement[case.get('element', 'FLARE')]
    p.flare.lens = _lens(surfaces)
    p.flare.light.position = QPointF(LIGHTS[surfaces][0] + float(move[0]), LIGHTS[surfaces][1] + float(move[1]))
    p.flare.ghost_aperture = Aperture(shape=ApertureShape(size=QSizeF(0.75, 0.75), blades=8, softness=0.1,
                                                          rotation=rotation))
    p.flare.ghost.fstop = fstop
    r = p.render
    r.resolution = QSize(case.get('width', 512), case.get('height', 512))
    r.grid_count = case.get('grid', 32)
    r.grid_length = 50.0 if surfaces == 50 else synthetic.GRID_LENGTH
    r.anti_aliasing = case.get('aa', 1)
    r.wavelength_sub_count = case.get('sub', 1)
    r.wavelength_count = case.get('wavelengths', 1)
    r.ghost.resolution = QSize(case.get('ghost_w', 256), case.get('ghost_h', 256))
    if surfaces == 50:  # the zoom: the reference's own wavelengths and ghost culling
        r.cull_percentage = 0.5
        p.flare.light.intensity = 0.1
    else:
        r.wavelengths = _wavelengths(case.get('spectra', r.wavelength_count))
    if 'star_w' in case:
        r.starburst.resolution = QSize(case['star_w'], case['star_h'])
        r.starburst.samples = case['samples']
        s = p.flare.starburst
        s.blur, s.rotation = case.get('blur', 0.0), case.get('rotation', 0.0)
        s.per_wavelength = case.get('spectra', 1) > 1
        s.vignetting_enabled = surfaces == 50
        dust = ApertureDust(strength=1.0, blur_sigma=2.0, seed=dust_seed) if case.get('dust') else ApertureDust()
        p.flare.starburst_aperture = Aperture(
            shape=ApertureShape(size=QSizeF(0.75, 0.75), blades=8, softness=0.05, rotation=rotation), dust=dust)
    return p


def _batch_projects(case: dict, seed: int) -> list:
    """A batch's frames: the lenses in turn, each with its own light."""
    return [_project(dict(case, lens=(8, 16, 24)[i % 3]), seed * 101 + i) for i in range(case['frames'])]


def _ghost(project: Project) -> Image:
    return GhostTask().run(project, GhostApertureTask().run(project))


def _target(case: dict, seed: int) -> torch.Tensor:
    """The image an adjoint case is fitted to: a smooth one of the flare's magnitude."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    coarse = torch.rand(1, 4, 8, 8, generator=g, device=DEVICE)
    size = (case['height'], case['width'])
    return torch.nn.functional.interpolate(coarse, size=size, mode='bilinear')[0].permute(1, 2, 0).contiguous()


def prepare(case: dict, seed: int) -> dict:
    kind = case['kind']
    if kind == 'batch':
        renderer = BatchRenderer(_batch_projects(case, seed))
        renderer.run()
        renderer.capture()
        return dict(kind=kind, renderer=renderer)
    project = _project(case, seed)
    if kind == 'render':
        return dict(kind=kind, project=project, engine=Engine(cache=False))
    if kind == 'trace':
        return dict(kind=kind, project=project, task=RaytracingTask(cache=False, accurate=case.get('accurate', False)))
    if kind == 'raster':
        return dict(kind=kind, project=project, rays=RaytracingTask(cache=False).run(project), ghost=_ghost(project),
                    task=RasterizingTask())
    n = len(project.flare.lens.lens_model.lens_elements) + 1
    project.flare.lens.coating_thickness = (550.0 / (4 * 1.38),) * n
    renderer = DifferentiableRenderer(project, _ghost(project).tensor)
    parameters = [t.to(torch.float32).requires_grad_(True) for t in renderer.params.tensors()]
    return dict(kind=kind, renderer=renderer, parameters=parameters, target=_target(case, seed))


def run(state: dict):
    kind = state['kind']
    if kind == 'render':
        if not state['engine'].render(state['project']):
            raise RuntimeError('the engine refused the project')
        return state['engine'].image.tensor
    if kind == 'batch':
        state['renderer'].replay()
        return state['renderer'].images
    if kind == 'trace':
        rays = state['task'].run(state['project']).tensor
        return dict(position=rays[0:2], aperture=rays[2:4], rrel=rays[4], reflectance=rays[5])
    if kind == 'raster':
        return state['task'].run(state['project'], state['rays'], state['ghost']).tensor
    # the optimiser holds float32 parameters; the lens geometry is evaluated from them in double
    image = state['renderer'].render(*[p.double() for p in state['parameters']])
    loss = ((image - state['target'])[..., :3] ** 2).mean()
    return dict(image=image.detach(), gradients=list(torch.autograd.grad(loss, state['parameters'])))


# ------------------------------------------------------------------------------ work
def _frames(case: dict) -> list:
    if case['kind'] == 'batch':
        return [dict(case, kind='render', element='FLARE', lens=(8, 16, 24)[i % 3]) for i in range(case['frames'])]
    return [case]


def _rays(case: dict) -> int:
    return sum(GHOSTS[c['lens']] * c['wavelengths'] * c['grid'] ** 2 for c in _frames(case) if 'lens' in c)


def _fragments(case: dict) -> int:
    """Shaded fragments: a ghost's quads together cover about one image area per wavelength pair
    (1.03 on the production frame), a third of it on the zoom and the 8-surface lens."""
    n = 0.0
    for c in _frames(case):
        if c['kind'] == 'trace' or 'lens' not in c:
            continue
        share = 1.0 if c['lens'] in (16, 24) else 0.33
        sub = c.get('sub', 1) if c['wavelengths'] > 1 else 1
        n += share * GHOSTS[c['lens']] * max(c['wavelengths'] - 1, 1) * sub * c['width'] * c['height']
    return int(n)


def work(case: dict) -> dict:
    kind, nbytes, flops = case['kind'], 0.0, 0.0
    if kind != 'raster':  # about 1.8 steps per element: there, back between the bounces, on
        flops += sum(_rays(c) * 1.8 * ELEMENTS[c['lens']] * INTERACTION_FLOPS for c in _frames(case) if 'lens' in c)
    flops += _fragments(case) * FRAGMENT_FLOPS * (3 if kind == 'adjoint' else 1)
    if kind in ('raster', 'trace'):
        nbytes += 24 * _rays(case)
    if kind == 'adjoint':
        nbytes += 16 * case['width'] * case['height']
    if case.get('element') == 'GHOST':  # three transforms of 5 n log2 n
        n = case['ghost_w'] * case['ghost_h']
        nbytes += 4 * n
        flops += 3 * 5 * n * math.log2(n)
    elif kind != 'trace':
        nbytes += 16 * sum(c['width'] * c['height'] for c in _frames(case))
    if 'star_w' in case:  # per sample: a position and a bilinear lookup; jitter adds two hashes
        n = case['star_w'] * case['star_h']
        flops += case.get('spectra', 1) * 5 * n * math.log2(n)
        flops += case['width'] * case['height'] * case['samples'] * (60 if case.get('blur') else 25)
        nbytes += 4 * n
    return dict(bytes=nbytes, flops=flops)


# ------------------------------------------------------------------------------ 64 bits
def exact(case: dict, seed: int):
    """The outputs in 64 bits from the same inputs, where that takes seconds; None elsewhere (whole
    frames of a size, batches, gradients; jittered starbursts, whose hash has no 64-bit value)."""
    kind = case['kind']
    project = _project(case, seed)
    if kind == 'trace':
        r = _trace64(project)
        return dict(position=r[0:2], aperture=r[2:4], rrel=r[4], reflectance=r[5])
    if kind == 'raster' and _fragments(case) * case.get('aa', 1) < 1e8:
        rays = RaytracingTask(cache=False).run(project).tensor
        return _raster64(project, rays.double(), _ghost(project).tensor.double())
    if kind != 'render':
        return None
    if case['element'] == 'GHOST':
        return _ghost64(project)
    if case['element'] == 'STARBURST' and not case.get('blur') and not case.get('rotation'):
        return _starburst64(project)
    if case['element'] == 'FLARE' and _fragments(case) * case.get('aa', 1) < 1e7:
        return _raster64(project, _trace64(project), _ghost64(project))
    return None


def _f64(x) -> torch.Tensor:
    return torch.as_tensor(np.asarray(x), device=DEVICE).double()


def _smoothstep(e0: float, e1: float, x: torch.Tensor) -> torch.Tensor:
    t = ((x - e0) / (e1 - e0)).nan_to_num(0.0, 1.0, 0.0).clamp(0, 1)
    return t * t * (3 - 2 * t)


def _ap1(xyz: torch.Tensor) -> torch.Tensor:
    m = _f64([[1.6410233797, -0.3248032942, -0.2364246952], [-0.6636628587, 1.6153315917, 0.0167563477],
              [0.0117218943, -0.0082844420, 0.9883948585]])
    return torch.cat([xyz @ m.T, torch.zeros_like(xyz[..., :1])], -1)


def _bilinear(tex: torch.Tensor, u: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """tex (h, w) at texel coordinates, 0 outside it."""
    h, w = tex.shape
    ok = torch.isfinite(u) & torch.isfinite(v)
    u, v = torch.where(ok, u, -9.0).clamp(-9, w + 9), torch.where(ok, v, -9.0).clamp(-9, h + 9)
    i, j = u.floor(), v.floor()
    a, b = u - i, v - j
    i, j = i.long(), j.long()

    def at(y, x):
        inside = (x >= 0) & (x < w) & (y >= 0) & (y < h)
        return torch.where(inside, tex[y.clamp(0, h - 1), x.clamp(0, w - 1)], 0.0)

    return ((1 - a) * (1 - b) * at(j, i) + a * (1 - b) * at(j, i + 1) + (1 - a) * b * at(j + 1, i)
            + a * b * at(j + 1, i + 1))


def _ndc(n: int) -> torch.Tensor:
    return 2 * torch.arange(n, device=DEVICE, dtype=torch.float64) / (n - 1) - 1


def _aperture64(aperture: Aperture, w: int, h: int) -> torch.Tensor:
    s = aperture.shape
    x, y = (_ndc(w) / s.size.width())[None, :], (_ndc(h) / s.size.height())[:, None]
    c, sn = math.cos(math.radians(s.rotation)), math.sin(math.radians(s.rotation))
    x, y = x * c + y * sn, y * c - x * sn
    sdf = torch.zeros_like(x)
    for i in range(s.blades):
        angle = (i / s.blades + 0.25) * 2 * math.pi
        sdf = torch.maximum(sdf, math.cos(angle) * x + math.sin(angle) * y)
    soft = s.softness / 10
    image = 1 - _smoothstep(1 - soft, 1 + soft, sdf)
    d = aperture.dust
    if d.strength > 0:
        noise = np.random.Generator(np.random.PCG64(d.seed)).random((h, w), dtype=np.float32)
        r = math.ceil(d.blur_sigma * 4)
        k = torch.exp(-torch.arange(-r, r + 1, device=DEVICE, dtype=torch.float64) ** 2 / (2 * d.blur_sigma ** 2))
        k = (k / k.sum()).view(1, 1, 1, -1)
        z = torch.nn.functional.pad(_f64(noise)[None, None], (r, r, r, r), mode='replicate')
        z = torch.nn.functional.conv2d(torch.nn.functional.conv2d(z, k), k.transpose(2, 3))[0, 0]
        image = image * (1 - d.strength * z)
    return image


def _fold(n: int) -> torch.Tensor:
    """0, 1, ... then the negative offsets: the chirp's coordinate along an axis of n."""
    i = torch.arange(n, device=DEVICE, dtype=torch.float64)
    return torch.where(i < n // 2, i, i - n)


def _ghost64(project: Project) -> torch.Tensor:
    """|frft(aperture)|: the fractional Fourier transform by chirp convolution."""
    size = project.render.ghost.resolution
    w, h = size.width(), size.height()
    z = torch.fft.fftshift(_aperture64(project.flare.ghost_aperture, w, h)).to(torch.complex128)
    alpha = 0.15 * (560 / 400) * (project.flare.ghost.fstop / 18)  # below 0.5 for every f-stop here
    z = torch.fft.ifftn(z, norm='ortho')
    phi = (alpha + 1) * math.pi / 2
    cot = 1 / math.tan(phi)
    sq = math.sqrt(1 + cot * cot)
    rows, cols = _fold(h), _fold(w)
    r = math.pi * (rows[:, None] ** 2 / h + cols[None, :] ** 2 / w)
    chirp = lambda c: torch.polar(torch.ones_like(r), r * c)  # noqa: E731
    f = torch.fft.fftn(chirp(sq), norm='ortho') * torch.fft.fftn(chirp(cot - sq) * z, norm='ortho')
    z = chirp(cot - sq) * torch.fft.ifftn(f, norm='ortho') * (abs(1 - 1j * cot) ** 0.5 / math.sqrt(w * h))
    return torch.fft.fftshift(z).abs() * math.sqrt(w * h)


def _starburst64(project: Project) -> torch.Tensor:
    config, r = project.flare.starburst, project.render
    aw, ah = r.starburst.resolution.width(), r.starburst.resolution.height()
    wl = [float(v) for v in r.wavelengths] if config.per_wavelength else [560.0]
    aperture = _aperture64(project.flare.starburst_aperture, aw, ah)
    r2 = _ndc(aw)[None, :] ** 2 + _ndc(ah)[:, None] ** 2
    spectra = []
    for lam in wl:
        chirp = torch.polar(torch.ones_like(r2), math.pi * r2 / (lam * 1e-6 * config.distance * 1e3))
        spectra.append(torch.fft.fftshift(torch.fft.fft2(aperture * chirp)).abs() ** 2)
    w, h = r.resolution.width(), r.resolution.height()
    pos = project.flare.light.position
    x = ((_ndc(w) - pos.x()) / config.scale.width())[None, :].expand(h, w)
    y = ((_ndc(h) + pos.y()) / (config.scale.height() * w / h))[:, None].expand(h, w)
    light = _f64(light_spectrum())
    acc = torch.zeros(h, w, 3, device=DEVICE, dtype=torch.float64)
    step_nm = (wl[-1] - wl[0]) / (len(wl) - 1) if len(wl) > 1 else 1.0
    for t in range(r.starburst.samples):
        s = t / r.starburst.samples
        lam = np.float32(s) * np.float32(340) + np.float32(390)  # a tie between two spectra is decided in 32 bits
        k = math.floor((np.float32(lam) - np.float32(wl[0])) / np.float32(step_nm) + np.float32(0.5))
        k = min(max(int(k), 0), len(wl) - 1)
        scale = (s * 340 + 390) / 560
        f = _bilinear(spectra[k], (x / scale * 0.5 + 0.5) * aw - 0.5, (y / scale * 0.5 + 0.5) * ah - 0.5)
        u = s * light.shape[0] - 0.5
        i, a = math.floor(u), u - math.floor(u)
        row = sum((wt * light[j, :3] for j, wt in ((i, 1 - a), (i + 1, a)) if 0 <= j < light.shape[0]),
                  torch.zeros(3, device=DEVICE, dtype=torch.float64))
        acc += 0.5 * row * f[..., None]  # the table's one row is sampled at its edge: half weight
    return _ap1(acc / r.starburst.samples * (config.intensity * 1e-6))


def _trace64(project: Project) -> torch.Tensor:
    """The six ray planes [6, P * W * G^2]: every path's rays stepped through its elements."""
    ti = host.trace_inputs(project)
    a = ti.args
    P, W, G, E = a.path_count, a.wavelength_count, a.grid_count, a.element_count
    el = {k: _f64(ti.elements[k]) for k in ('radius', 'center', 'height', 'ior')}
    layers, coating = ti.elements['coating_layers'], ti.elements['coating']
    thickness, coef = ti.elements['coating_thickness'].astype(np.float64), _f64(ti.elements['coefficients'])
    wl = _f64(ti.wavelengths)
    l2 = (wl[:, None] * 1e-3) ** 2
    n2 = 1 + sum(coef[None, :, 2 * k] * l2 / (l2 - coef[None, :, 2 * k + 1]) for k in range(3))
    ior = torch.where((el['ior'] > 1)[None, :], n2.clamp_min(0).sqrt(), el['ior'][None, :])  # [W, E]
    g = a.grid_length * (torch.arange(G, device=DEVICE, dtype=torch.float64) / (G - 1) - 0.5)
    gx, gy = g.repeat(G), g.repeat_interleave(G)
    v = -_f64([a.direction[0], a.direction[1], a.direction[2]])
    light = v / v.norm()
    out = torch.empty(6, P, W, G * G, device=DEVICE, dtype=torch.float64)

    def hit(p, d, e):
        radius, cz = float(el['radius'][e]), -float(el['center'][e])
        if radius == 0:
            q = p + d * ((cz - p[2]) / d[2])
            normal = torch.zeros_like(p)
            normal[2] = torch.where(d[2] < 0, 1.0, -1.0)
            return q, normal, d[2] != 0
        u = -p.clone()
        u[2] += cz
        u1 = d * (u * d).sum(0)
        dist = (u - u1).pow(2).sum(0).sqrt()
        sgn = torch.where(radius * d[2] > 0, -1.0, 1.0)
        m = (radius * radius - dist * dist).clamp_min(0).sqrt()
        q = p + u1 - d * m * sgn
        normal = q.clone()
        normal[2] -= cz
        return q, normal / normal.norm(dim=0) * sgn, (dist <= abs(radius)) & (d[2] != 0)

    p0 = torch.stack([gx, -gy, torch.ones_like(gx)])
    q0, _, ok0 = hit(p0, torch.tensor([0.0, 0.0, -1.0], device=DEVICE, dtype=torch.float64)[:, None].expand_as(p0), 0)
    start = torch.where(ok0, q0, 0.0) - light[:, None]
    for path, (b1, b2) in enumerate(ti.paths.tolist()):
        pos = start[:, None, :].expand(3, W, G * G).clone()
        d = light[:, None, None].expand(3, W, G * G).clone()
        alive = torch.ones(W, G * G, device=DEVICE, dtype=torch.bool)
        apt, rrel = torch.zeros_like(pos[:2]), torch.zeros_like(pos[0])
        refl = torch.ones_like(rrel)
        i, step, delta = 0, 0, 1
        while 0 <= i < E:
            q, n, ok = hit(pos, d, i)
            alive = alive & ok
            pos = torch.where(alive, q, pos)
            height = float(el['height'][i])
            if i == a.aperture_index:
                apt = torch.where(alive, q[:2] / height, apt)
            else:
                rrel = torch.where(alive, torch.maximum(rrel, q[:2].norm(dim=0) / height), rrel)
                if i < E - 1:
                    forward = d[2] >= 0
                    after = ior[:, i + 1][:, None] if i + 1 < E else torch.ones_like(ior[:, :1])
                    before = ior[:, i - 1][:, None] if i > 0 else torch.ones_like(ior[:, :1])
                    na, nb = torch.where(forward, after, before), ior[:, i][:, None].expand_as(rrel)
                    c = -(d * n).sum(0)
                    if (step == 0 and i == b1) or (step == 1 and i == b2):
                        step, delta = step + 1, -delta
                        R = _reflectance(torch.acos(c.clamp(-1, 1)) + 1e-9, wl[:, None], na, nb, int(layers[i]),
                                         float(coating[i]), thickness[i], a)
                        refl = torch.where(alive & (R > 0), refl * R, refl)
                        d = torch.where(alive, d + n * 2 * c, d)
                    else:
                        o = na / nb
                        s2 = o * o * (1 - c * c)
                        t = (o * d + (o * c - (1 - s2).abs().sqrt()) * n) * (s2 < 1)
                        d = torch.where(alive, t, d)
                        alive = alive & (d[2] != 0)
            i += delta
        out[0:2, path], out[2:4, path], out[4, path] = pos[:2], apt, rrel
        out[5, path] = torch.where(alive, refl, math.nan)
    return out.view(6, -1)


def _reflectance(th, lam, n0, n2, layers, coating, thickness, a):
    sin, cos, tan, asin = torch.sin, torch.cos, torch.tan, torch.asin
    if layers == 2:
        na, nb = a.coating_layer_ior[0], a.coating_layer_ior[1]
        s0, c0 = sin(th), cos(th)
        ca, cb, c2 = (torch.sqrt(1 - (n0 * s0 / m) ** 2) for m in (na, nb, n2))
        d1, d2 = (4 * math.pi / lam * m * t * c for m, t, c in ((na, thickness[0], ca), (nb, thickness[1], cb)))
        e1, e2 = torch.polar(torch.ones_like(d1), d1), torch.polar(torch.ones_like(d2), d2)
        total = 0
        media = ((n0, c0), (na, ca), (nb, cb), (n2, c2))
        for swap in (False, True):
            r = []
            for (ni, ci), (nj, cj) in zip(media[:-1], media[1:]):
                p, q = (nj * ci, ni * cj) if swap else (ni * ci, nj * cj)
                r.append((p - q) / (p + q))
            inner = (r[1] + r[2] * e2) / (1 + r[1] * r[2] * e2)
            total = total + ((r[0] + inner * e1) / (1 + r[0] * inner * e1)).abs() ** 2
        return total / 2
    if layers == 1 or coating > 0:
        n1 = (n0 * n2).sqrt().clamp_min(a.coating_min_ior)
        d1 = thickness[0] if layers == 1 else coating / (4 * n1)
        t1, t2 = asin(sin(th) * n0 / n1), asin(sin(th) * n0 / n2)
        rs01, rp01 = -sin(th - t1) / sin(th + t1), tan(th - t1) / tan(th + t1)
        ts01 = 2 * sin(t1) * cos(th) / sin(th + t1)
        tp01 = ts01 * cos(th - t1)
        ris = ts01 ** 2 * -sin(t1 - t2) / sin(t1 + t2)
        rip = tp01 ** 2 * tan(t1 - t2) / tan(t1 + t2)
        dy = d1 * n1
        dx = tan(t1) * dy
        c = cos(4 * math.pi / lam * ((dx * dx + dy * dy).sqrt() - dx * sin(th)))
        return (rs01 ** 2 + ris ** 2 + 2 * rs01 * ris * c + rp01 ** 2 + rip ** 2 + 2 * rp01 * rip * c) / 2
    t1 = asin(sin(th) * n0 / n2)
    rs = (n0 * cos(th) - n2 * cos(t1)) / (n0 * cos(th) + n2 * cos(t1))
    rp = (n0 * cos(t1) - n2 * cos(th)) / (n0 * cos(t1) + n2 * cos(th))
    return (rs * rs + rp * rp) / 2


SAMPLES = (0, 1, 0, 1, 2, 0, 3, 4, 1, 6, 2, 5, 0, 3, 7)  # the n-rook rows of 1, 2, 4 and 8 samples


def _raster64(project: Project, rays: torch.Tensor, ghost: torch.Tensor) -> torch.Tensor:
    """The raster of given rays: quads, vertices, integer coverage and mean-value shading of every
    covered pixel, each fragment added to its pixel in 64 bits."""
    a = host.raster_args(project, 0, len(project.render.wavelengths), tuple(ghost.shape))
    W, WS, S, G = a.wavelength_count, a.wavelength_sub_count, a.sub_steps, a.grid_count
    width, height, B = a.width, a.height, a.bin_size
    area0, min_area = host.quad_constants(project)
    r = rays.view(6, -1, W, G, G)
    P = r.shape[1]
    px, py, refl = r[0], r[1], r[5]
    corner = lambda z: torch.stack([z[..., :-1, :-1], z[..., :-1, 1:], z[..., 1:, 1:], z[..., 1:, :-1]], -1)  # noqa: E731
    cx, cy, crr = corner(px), corner(py), corner(r[4])
    valid = ~corner(refl).isnan()
    count = valid.sum(-1)
    order = torch.sort((~valid).to(torch.int8), dim=-1, stable=True).indices  # valid corners first
    vx, vy = cx.gather(-1, order), cy.gather(-1, order)
    three = count == 3
    vx[..., 3], vy[..., 3] = torch.where(three, vx[..., 2], vx[..., 3]), torch.where(three, vy[..., 2], vy[..., 3])
    crr[..., 3] = torch.where(three, crr[..., 2], crr[..., 3])

    def tri(i, j, k):
        return ((vx[..., i] - vx[..., j]) * (vy[..., k] - vy[..., i])
                - (vy[..., i] - vy[..., j]) * (vx[..., k] - vx[..., i]))

    area = torch.where(three, tri(0, 1, 2).abs(), (tri(0, 1, 2) + tri(0, 2, 3)).abs() / 2).clamp_min(min_area)
    alive = torch.cumprod((count >= 3).to(torch.int8), dim=1).bool()  # a bad wavelength ends the quad
    inten = torch.where(alive, area0 / area, 0.0)  # [P, W, G-1, G-1]
    drawn = alive[:, -1] & ~(crr > 1).all(-1).all(1)
    # vertices: the mean of the positive intensities around them (neighbours by flat index)
    flat = inten.reshape(P, W, -1)
    Q = (G - 1) ** 2
    yy, xx = torch.meshgrid(torch.arange(G, device=DEVICE), torch.arange(G, device=DEVICE), indexing='ij')
    total, hits = torch.zeros(P, W, G, G, device=DEVICE, dtype=torch.float64), 0
    for dy, dx in ((-1, -1), (-1, 0), (0, -1), (0, 0)):
        nb = (yy + dy) * (G - 1) + xx + dx
        z = torch.where((nb >= 0) & (nb < Q), flat[..., nb.clamp(0, Q - 1)], 0.0)
        total, hits = total + z, hits + (z > 0)
    ok = ~refl.isnan()
    vint = total / hits.clamp_min(1)
    st = float(a.screen_transform)
    attrs = torch.stack([px * st + width / 2, py * st + height / 2, r[2], r[3], r[4], refl, vint])  # [7, P, W, G, G]
    ok_quad = corner(ok).all(-1)
    # a pair's far end: the next wavelength, or with one wavelength the next vertex in memory
    # (blended with weight 0, yet an invalid one drops the pair; a valid zero vertex follows the last)
    after = torch.cat([ok.flatten()[1:], ok.new_ones(1)]).view(ok.shape)
    end_ok = ok_quad[:, 1:] if W > 1 else corner(after).all(-1)
    bins = []
    for lo, hi, half, n in ((vx.amin((1, -1)), vx.amax((1, -1)), width // 2, width),
                            (vy.amin((1, -1)), vy.amax((1, -1)), height // 2, height)):
        s0, s1 = (torch.trunc((z * st).nan_to_num(0.0).clamp(-2e9, 2e9)).long() + half for z in (lo, hi))
        last = (n + B - 1) // B - 1
        bins.append((torch.div(s0 - 1, B, rounding_mode='floor').clamp_min(0),
                     torch.div(s1, B, rounding_mode='floor').clamp_max(last)))
    spectrum = _f64(light_spectrum())[:, :3]
    rgb = torch.zeros(height * width, 3, device=DEVICE, dtype=torch.float64)
    gh, gw = ghost.shape
    for w in range(max(W - 1, 1)):
        w1 = min(w + 1, W - 1)
        for i in range(WS):
            t = i / WS
            m = attrs[:, :, w] + (attrs[:, :, w1] - attrs[:, :, w]) * t
            keep = drawn & ok_quad[:, w] & end_ok[:, w]
            rec = corner(m).permute(1, 2, 3, 0, 4)[keep]  # [n, 7, 4]
            rect = [z[keep] for pair in bins for z in pair]
            colour = torch.ones(3, device=DEVICE, dtype=torch.float64)
            if W > 1:
                u = (w + 0.5 + i / WS) / W * spectrum.shape[0] - 0.5
                j, f = math.floor(u), u - math.floor(u)
                at = lambda k: spectrum[min(max(k, 0), spectrum.shape[0] - 1)]  # noqa: E731
                colour = (1 - f) * at(j) + f * at(j + 1)
            _shade64(rgb, rec, rect, colour, ghost, a, gw, gh)
    rgb = rgb * (float(a.intensity) / (W * S * WS))
    image = _ap1(torch.where((rgb > 0).any(-1, keepdim=True), rgb, 0.0))
    return image.view(height, width, 4).flip(0)


def _shade64(rgb, rec, rect, colour, ghost, a, gw, gh):
    """Adds records [n, 7, 4] (x, y, u, v, rrel, reflectance, intensity of the four corners)."""
    S, B, width, height = a.sub_steps, a.bin_size, a.width, a.height
    q = torch.trunc((rec[:, :2] * S).clamp(-2147483648, 2147483647)).long()  # [n, 2, 4]
    lo = torch.div(q.amin(-1), S, rounding_mode='floor') - 1
    hi = torch.div(q.amax(-1), S, rounding_mode='floor') + 1
    far = (q.abs() > 16382).any(-1).any(-1)  # 32-bit edge functions may wrap: every pixel of its bins
    bx0, bx1, by0, by1 = rect
    x0, x1 = torch.where(far, bx0 * B, torch.maximum(lo[:, 0], bx0 * B)), torch.where(
        far, bx1 * B + B - 1, torch.minimum(hi[:, 0], bx1 * B + B - 1)).clamp_max(width - 1)
    y0, y1 = torch.where(far, by0 * B, torch.maximum(lo[:, 1], by0 * B)), torch.where(
        far, by1 * B + B - 1, torch.minimum(hi[:, 1], by1 * B + B - 1)).clamp_max(height - 1)
    nx, ny = (x1 - x0 + 1).clamp_min(0), (y1 - y0 + 1).clamp_min(0)
    pixels = nx * ny
    ends = pixels.cumsum(0)
    begin, n = 0, len(pixels)
    while begin < n:
        base = int(ends[begin - 1]) if begin else 0
        end = int(torch.searchsorted(ends, base + (1 << 22)).clamp(begin + 1, n))
        k = torch.repeat_interleave(torch.arange(begin, end, device=DEVICE), pixels[begin:end])
        o = torch.arange(len(k), device=DEVICE) + base - (ends - pixels)[k]
        x, y = x0[k] + o % nx[k], y0[k] + torch.div(o, nx[k], rounding_mode='floor')
        begin = end
        hits = torch.zeros_like(x)
        for s in range(S):
            hits += _inside64(q[k], x * S + s, y * S + SAMPLES[S - 1 + s])
        sel = hits > 0
        k, x, y, hits = k[sel], x[sel], y[sel], hits[sel]
        if not len(k):
            continue
        wt = _weights64(q[k], x * S + S // 2, y * S + S // 2)
        z = (rec[k] * wt[:, None, :]).sum(-1)
        u = ((z[:, 2] / a.ghost_scale + 1) / 2) * gw - 0.5
        v = ((z[:, 3] / a.ghost_scale + 1) / 2) * gh - 0.5
        f = _bilinear(ghost, u, v) * _smoothstep(1.0, 0.95, z[:, 4]) * z[:, 5].clamp_min(0) * z[:, 6].clamp_min(0)
        rgb.index_add_(0, y * width + x, (f * hits)[:, None] * colour)


def _inside64(q, x, y):
    """The reference's quad test: five 32-bit edge functions with the top-left rule."""
    wrap = lambda z: torch.remainder(z + 2147483648, 4294967296) - 2147483648  # noqa: E731

    def edge(i, j):
        ax, ay, bx, by = q[:, 0, i], q[:, 1, i], q[:, 0, j], q[:, 1, j]
        ex, ey = bx - ax, by - ay
        bias = torch.where(((ey == 0) & (ex > 0)) | (ey > 0), 0, -1)
        return wrap((ax - bx) * (y - ay) - (ay - by) * (x - ax) + bias) >= 0

    def area(i, j, k):
        return wrap((q[:, 0, i] - q[:, 0, j]) * (q[:, 1, k] - q[:, 1, i])
                    - (q[:, 1, i] - q[:, 1, j]) * (q[:, 0, k] - q[:, 0, i]))

    w01, w12, w23, w30, w20 = edge(0, 1), edge(1, 2), edge(2, 3), edge(3, 0), edge(2, 0)
    front = (w20 & w01 & w12 & (w23 | w30)) | (~w20 & w23 & w30 & (w01 | w12))
    back = (~w20 & ~w01 & ~w12 & (~w23 | ~w30)) | (w20 & ~w23 & ~w30 & (~w01 | ~w12))
    return (front | back) & ~((area(0, 1, 2) == 0) & (area(0, 2, 3) == 0))


def _weights64(q, x, y):
    """Mean-value coordinates of the sample point in the integer quad."""
    s = q.double() - torch.stack([x, y], 1)[..., None]
    n = s.roll(-1, -1)
    cross = s[:, 0] * n[:, 1] - n[:, 0] * s[:, 1]
    length = s.norm(dim=1)
    t = (length * length.roll(-1, -1) - (s * n).sum(1)) / torch.where(cross == 0, 1e-3, cross)
    w = (t.roll(1, -1) + t) / length
    w = w / w.sum(-1, keepdim=True)
    on = length == 0
    first = on & (on.cumsum(-1) == 1)
    return torch.where(on.any(-1, keepdim=True), first.double(), w)
