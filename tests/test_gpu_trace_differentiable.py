"""The forward traces of a differentiated render: everything but the reflectance is that of rf_trace and
rf_trace_accurate bit for bit, and the reflectances have the form that the adjoint differentiates, in both. Where the
geometry is exact in FP32 (flat elements, light along the axis, no dispersion) the two therefore agree bit for bit."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import reduced  # noqa: E402
from test_gpu_trace_paths import same_bits  # noqa: E402

from realflare_gb300 import prepare  # noqa: E402
from realflare_gb300._abi import check, lib  # noqa: E402
from realflare_gb300.device import empty, ptr, stream_handle, to_device  # noqa: E402


def trace(name, elements, ti):
    el, pa, wl = to_device(elements.view(np.uint8)), to_device(ti.paths), to_device(ti.wavelengths)
    rays = empty((6, ti.ray_count))
    check(getattr(lib(), name)(ptr(el), ptr(pa), ptr(wl), ctypes.byref(ti.args), ptr(rays), stream_handle()), name)
    torch.cuda.synchronize()
    return rays


def coated(ti, two_layers):
    """The elements with every kind of coating among them."""
    el = ti.elements.copy()
    for i in range(len(el)):
        kind = i % (4 if two_layers else 3)
        el[i]['coating'] = 550 if kind == 1 else 0
        el[i]['coating_layers'] = (0, 0, 1, 2)[kind]
        el[i]['coating_thickness'] = (100.0, 80.0)
    ti.args.coating_layer_ior[0], ti.args.coating_layer_ior[1] = 1.38, 2.1
    return el


@pytest.mark.parametrize('two_layers', [False, True])
@pytest.mark.parametrize('workload,grid', [('plain-8', 33), ('spectral-16', 24)])
@pytest.mark.parametrize('plain,differentiable', [('rf_trace', 'rf_trace_differentiable'),
                                                  ('rf_trace_accurate', 'rf_trace_accurate_differentiable')])
def test_other_outputs(plain, differentiable, workload, grid, two_layers):
    ti = prepare.trace_inputs(reduced(workload, grid=grid, wavelengths=3).project)
    el = coated(ti, two_layers)
    a, b = trace(plain, el, ti), trace(differentiable, el, ti)
    assert same_bits(a[:5], b[:5])
    assert torch.equal(torch.isnan(a[5]), torch.isnan(b[5]))
    ok = ~torch.isnan(a[5])
    assert ok.any() and (a[5] - b[5])[ok].norm() <= 1e-4 * a[5][ok].norm()


@pytest.mark.parametrize('layers', [0, 2])
@pytest.mark.parametrize('plain,differentiable', [('rf_trace', 'rf_trace_differentiable'),
                                                  ('rf_trace_accurate', 'rf_trace_accurate_differentiable')])
def test_no_coating(plain, differentiable, layers):
    """Uncoated, and two layers without thickness: between equal indices (at the element before the stop) the reflectance
    is 0, which the trace does not multiply by, or a rounding residue, which it does; alike in both forms."""
    ti = prepare.trace_inputs(reduced('spectral-16', grid=24, wavelengths=3).project)
    el = ti.elements.copy()
    el['coating'] = 0
    el['coating_layers'] = layers
    el['coating_thickness'] = 0.0
    ti.args.coating_layer_ior[0], ti.args.coating_layer_ior[1] = 1.38, 2.1
    a, b = trace(plain, el, ti), trace(differentiable, el, ti)
    ok = ~torch.isnan(a[5])
    assert ((a[5] < 1e-9) & ok).any()
    assert (a[5] - b[5])[ok].norm() <= 1e-4 * a[5][ok].norm()


@pytest.mark.parametrize('two_layers', [False, True])
def test_accurate_has_the_adjoints_reflectances(two_layers):
    ti = prepare.trace_inputs(reduced('spectral-16', grid=5, wavelengths=4).project)
    el = coated(ti, two_layers)
    el['center'] -= el['radius']
    el['radius'] = 0.0
    el[0]['coefficients'][0] = np.nan
    ti.args.direction[0], ti.args.direction[1], ti.args.direction[2] = 0.0, 0.0, 1.0
    a, b = trace('rf_trace_differentiable', el, ti), trace('rf_trace_accurate_differentiable', el, ti)
    assert not torch.isnan(a[5]).any() and (a[5] > 0).any()
    assert torch.equal(a[5], b[5])


def test_renderer_traces_with_it():
    from realflare_gb300.diff import DifferentiableRenderer

    w = reduced('differentiable-16', grid=12, resolution=64, paths=20, wavelengths=2)
    p = w.project
    p.flare.lens.coating_thickness = (100.0,) * (len(p.flare.lens.lens_model.lens_elements) + 1)
    r = DifferentiableRenderer(p, torch.ones((64, 64), device='cuda'), w.paths, accurate=True)
    rays, el, targs = r.trace_kernels(*r.params.elements(*r.params.tensors(), r.E))
    want = torch.empty_like(rays)
    check(lib().rf_trace_accurate_differentiable(el.data_ptr(), r.paths.data_ptr(), r.wavelengths.data_ptr(),
                                                 ctypes.byref(targs), want.data_ptr(), stream_handle()), 'trace')
    assert same_bits(rays, want)
