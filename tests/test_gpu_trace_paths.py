"""Paths traced together (shared legs) against the trace of each path alone, bit for bit: paths in any
order, repeated, without reflections, with reflections at the stop, at the last element, outside the lens."""

import copy
import ctypes

import numpy as np
import pytest
import torch

from realflare_gb300 import prepare, synthetic
from realflare_gb300._abi import check, lib
from realflare_gb300.device import empty, ptr, stream_handle, to_device

pytestmark = pytest.mark.gpu


def inputs(grid: int, wavelengths: int, count: int):
    p = copy.deepcopy(synthetic.workload('plain-8').project)
    p.render.grid_count = grid
    p.render.wavelength_count = wavelengths
    p.render.wavelengths = tuple(float(v) for v in np.linspace(390.0, 700.0, wavelengths))
    elements = prepare.trace_inputs(p).args.element_count
    every = [(a, b) for a in range(-1, elements + 2) for b in range(-1, elements + 2)]
    rng = np.random.default_rng(grid + count)
    lens_paths = [q for q in every if q[0] > q[1] >= 0]
    paths = [every[i] for i in rng.integers(len(every), size=count // 3)]
    paths += [lens_paths[i] for i in rng.integers(len(lens_paths), size=count - len(paths))]
    return prepare.trace_inputs(p, paths=[paths[i] for i in rng.permutation(count)])


def same_bits(a, b) -> bool:
    return torch.equal(torch.nan_to_num(a, nan=-7.0), torch.nan_to_num(b, nan=-7.0))


# blocks of 128 rays: 1, 2, 4, 8 and 16 paths a block, path counts that leave a short last block
@pytest.mark.parametrize('grid, wavelengths, count', [(2, 1, 1), (7, 3, 40), (33, 25, 23), (65, 12, 25), (129, 5, 31),
                                                      (129, 7, 47)])
def test_together_and_alone(grid, wavelengths, count):
    ti = inputs(grid, wavelengths, count)
    a = ti.args
    el, pa, wl = to_device(ti.elements.view(np.uint8)), to_device(ti.paths), to_device(ti.wavelengths)
    rays, alone = empty((6, ti.ray_count)), empty((6, ti.ray_count))
    steps = prepare.intersection_count(a.element_count)
    inter = empty((ti.ray_count, steps, 8))
    s = stream_handle()
    check(lib().rf_trace(ptr(el), ptr(pa), ptr(wl), ctypes.byref(a), ptr(rays), s), 'rf_trace')
    check(lib().rf_trace_intersections(ptr(el), ptr(pa), ptr(wl), ctypes.byref(a), ptr(alone), ptr(inter), steps, s),
          'rf_trace_intersections')
    assert same_bits(rays, alone)


@pytest.mark.parametrize('grid, wavelengths, count', [(9, 2, 13), (25, 9, 33), (33, 15, 61)])
def test_accurate_together_and_alone(grid, wavelengths, count):
    ti = inputs(grid, wavelengths, count)
    a = ti.args
    el, pa, wl = to_device(ti.elements.view(np.uint8)), to_device(ti.paths), to_device(ti.wavelengths)
    rays, one = empty((6, ti.ray_count)), empty((6, ti.ray_count // count))
    s = stream_handle()
    check(lib().rf_trace_accurate(ptr(el), ptr(pa), ptr(wl), ctypes.byref(a), ptr(rays), s), 'rf_trace_accurate')
    a.path_count = 1
    for k in range(count):
        check(lib().rf_trace_accurate(ptr(el), ptr(pa[k:]), ptr(wl), ctypes.byref(a), ptr(one), s), 'rf_trace_accurate')
        assert same_bits(rays.view(6, count, -1)[:, k], one)
