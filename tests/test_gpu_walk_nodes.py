"""The walks' half-precision nodes, relative to their domain, where that is hardest:
domains far from the origin or of extreme size, flat ones, and vertices that are not
finite.  The queue kernels, which read the exact boxes, give the image to match."""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from test_gpu_walks import _pair

pytestmark = pytest.mark.gpu

CFG = dict(image_w=61, image_h=47, ao_mode=0, ao_samples=2, pixel_samples=2, bounces=3)


def _mapped(scale, shift, edit=None):
    base = scenes.wavelet_grid(2, 24, colors="albedo", light="point")
    doms = []
    for k, d in enumerate(base.domains):
        v = (d.vertices.astype(np.float64) * scale + shift).astype(np.float32)
        bounds = np.concatenate([v.min(0), v.max(0)])
        if edit:
            edit(k, v)
        doms.append(sg.Domain(v, d.faces, d.colors, bounds))
    sc = sg.Scene(doms, [])
    sc.lights = scenes.make_lights("point+diffuse", *scenes.scene_box(sc))
    return sc


@pytest.mark.parametrize("scale,shift", [
    ((1, 1, 1), (1e4, -3e4, 2e4)), ((1, 1, 1), (1e6, 1e6, -1e6)),  # boxes of a few units in the last place
    ((1e3, 1e3, 1e3), (0, 0, 0)), ((1e6, 1e6, 1e6), (0, 0, 0)), ((0.05, 0.05, 0.05), (0, 0, 0)),
    ((1, 1, 0), (0, 0, 3)),                                        # flat domains
    ((100, 1, 0.01), (0, 0, 0)),
])
def test_placed_and_sized_domains(lib_built, scale, shift):
    sc = _mapped(np.array(scale, float), np.array(shift, float))
    _pair(sc, scenes.orbit_camera(sc), **CFG)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38])
def test_vertices_that_are_not_finite(lib_built, value):
    def edit(k, v):
        v[7 + k, k % 3] = value
        if k == 3:
            v[100] = value

    sc = _mapped(np.ones(3), np.zeros(3), edit)
    img, st = _pair(sc, scenes.orbit_camera(sc), **CFG)
    assert st["rays_shadow"] > 0
