"""The walks' half-precision nodes, relative to their domain, where that is hardest:
domains far from the origin or of extreme size, flat ones, and vertices that are not
finite.  The queue kernels, which read the exact boxes, give the image to match."""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config
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


def _routes(scene, cam):
    """A frame as the scene is traced by default and by one launch per depth bucket of the
    queues: the same image.  The nodes per visit of both."""
    out = []
    for launches in (0, 4):
        t = sg.Tracer(small_config(bucket_launches=launches, **CFG))
        t.set_scene(scene)
        t.set_camera(*cam)
        img, st = t.trace()
        assert st["rays_shadow"] > 0
        out.append((img.view(np.uint32), st["nodes_radiance"] / st["visits_radiance"]))
    assert np.array_equal(out[0][0], out[1][0])
    return out[0][1], out[1][1]


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_vertices_that_are_not_finite(lib_built, value):
    def edit(k, v):
        v[7 + k, k % 3] = value
        if k == 3:
            v[100] = value

    sc = _mapped(np.ones(3), np.zeros(3), edit)
    _routes(sc, scenes.orbit_camera(sc))


def _detail(scale, stray=None, domains=(0, 1, 2, 3, 4, 5, 6, 7)):
    """Surfaces of `scale` times their cell, each with a quad across the cell and, with
    `stray`, a triangle without area whose far end lies that far out.  Only in `domains`."""
    base = scenes.wavelet_grid(2, 40, colors="albedo", light="point")
    doms = []
    for k, d in enumerate(base.domains):
        lo, hi = d.bounds[:3], d.bounds[3:]
        here = scale if k in domains else 1.0
        v = (d.vertices - (lo + hi) / 2) * np.float32(here) + (lo + (hi - lo) * np.array([0.5, 0.4, 0.3], np.float32))
        quad = np.array([lo, [hi[0], lo[1], lo[2]], [hi[0], lo[1], hi[2]], [lo[0], lo[1], hi[2]]], np.float32)
        far = np.full((1, 3), stray if stray and k in domains else hi, np.float32)
        n = len(v)
        faces = [[n, n + 1, n + 2], [n, n + 2, n + 3], [n, n + 4, n + 4]]
        doms.append(sg.Domain(np.concatenate([v, quad, far]), np.concatenate([d.faces, faces]),
                              np.concatenate([d.colors, np.full(5, 0x808080, np.uint32)]), d.bounds))
    sc = sg.Scene(doms, [])
    sc.lights = scenes.make_lights("point", *scenes.scene_box(sc))
    small = doms[domains[0]].vertices[:-5]
    centre, size = small.mean(0), float(np.ptp(small, axis=0).max())
    at = centre + np.float32(1.2 * size) * np.array([0.5, 0.6, 1.0], np.float32)
    return sc, (at.astype(np.float32), centre.astype(np.float32), np.array([0, 1, 0], np.float32))


@pytest.mark.parametrize("scale,stray,domains", [
    (1.0, None, range(8)), (0.01, None, range(8)), (0.001, None, range(8)), (1e-4, None, [5]),
    (1.0, 1e3, range(8)), (1.0, 1e6, [2]), (1.0, 1e20, range(8)), (1.0, 3e38, [0, 7]),
])
def test_detail_far_smaller_than_its_domain(lib_built, scale, stray, domains):
    # nodes that half precision cannot hold apart are not walked: at most twice the
    # nodes a visit that exact boxes need
    sc, cam = _detail(scale, stray, list(domains))
    here, exact = _routes(sc, cam)
    assert here <= 2.0 * exact + 2.0, (here, exact)


def test_scenes_that_walk_and_do_not_in_turn(lib_built):
    cfg = small_config(**CFG)
    t = sg.Tracer(cfg)
    kept = []
    for scale in (1.0, 1e-4, 1.0, 1e-4, 1e-4, 1.0):
        sc, cam = _detail(scale)
        fresh = sg.Tracer(cfg)
        for x in (t, fresh):
            x.set_scene(sc)
            x.set_camera(*cam)
        want, st = fresh.trace()
        kept.append(st["kernel_launches"])
        for _ in range(3):
            assert np.array_equal(t.trace()[0].view(np.uint32), want.view(np.uint32))
    assert kept[0] == kept[2] == kept[5] < kept[1] == kept[3] == kept[4]  # walks need fewer
