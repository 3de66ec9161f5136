"""In-core frames whose rays walk their own domain lists against the queue kernels.

Frames without captures walk whole rays; bucket_launches = 4 keeps the
per-domain queues.  Both must give the same image bit for bit and list the same
(ray, domain) pairs, for domain counts around the sizes where the list pass
changes (no groups below 16 domains, groups of 4, 16 and 64, the hierarchy above), with boxes that touch, overlap, are flat or inverted, and with rays
parallel to their planes.
"""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config

pytestmark = pytest.mark.gpu


def bits(a):
    return a.view(np.uint32)


def _boxes_scene(n, seed, odd=False):
    """n boxes of 12 triangles on a jittered grid; every fifth one overlaps its neighbours."""
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n ** (1 / 3)))
    corners = np.array([[x, y, z] for z in (0, 1) for y in (0, 1) for x in (0, 1)], np.float32)
    quads = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    faces = np.array([t for a, b, c, d in quads for t in ((a, b, c), (a, c, d))], np.uint32)
    domains = []
    for d in range(n):
        cell = np.array([d % g, (d // g) % g, d // (g * g)], np.float32)
        size = np.float32(1.6 if d % 5 == 4 else 0.7)
        v = (cell + corners * size).astype(np.float32)
        bounds = np.concatenate([v.min(0), v.max(0)])
        if d % 2 == 0:
            bounds[3:] = np.maximum(bounds[3:], cell + 1)  # touches the next cell's plane
        if odd and d % 7 == 3:
            bounds[[1, 4]] = bounds[[4, 1]]  # inverted along y
        if odd and d % 7 == 5:
            v[:, 2] = v[0, 2]  # flat
            bounds = np.concatenate([v.min(0), v.max(0)])
        colour = int(rng.integers(1 << 24))
        domains.append(sg.Domain(v, faces, np.full(8, colour, np.uint32), bounds))
    sc = sg.Scene(domains, [])
    sc.lights = scenes.make_lights("point+diffuse", *scenes.scene_box(sc))
    return sc


def _pair(scene, cam, **cfg):
    out = []
    for launches in (0, 4):
        t = sg.Tracer(small_config(bucket_launches=launches, **cfg))
        t.set_scene(scene)
        t.set_camera(*cam)
        img, st = t.trace()
        again, st2 = t.trace()
        assert np.array_equal(bits(img), bits(again))
        out.append((img, st, st2))
    (a, sa, sa2), (b, sb, _) = out
    assert np.array_equal(bits(a), bits(b))
    for k in ("rays_primary", "rays_shadow", "rays_bounce"):
        assert sa[k] == sb[k]
    assert sa["visits_radiance"] + sa["visits_culled"] == sb["visits_radiance"] + sb["visits_culled"]
    assert sa["visits_radiance"] <= sb["visits_radiance"]
    for k in ("visits_radiance", "visits_shadow", "nodes_radiance", "tris_shadow"):
        assert sa[k] == sa2[k]  # a ray's own order repeats exactly
    return a, sa


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 130, 1024, 1030])
@pytest.mark.parametrize("ao", [0, 1])
def test_walks_equal_queues(lib_built, n, ao):
    sc = _boxes_scene(n, n, odd=True)
    cam = scenes.orbit_camera(sc)
    cfg = dict(image_w=61, image_h=47, ao_mode=ao, ao_samples=3, pixel_samples=2, bounces=1 if ao else 4, list_size=32)
    img, st = _pair(sc, cam, **cfg)
    assert st["rays_shadow"] > 0 and img[..., :3].max() > 0


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (31, 1, 1), (33, 5, 3), (640, 360, 1)])
def test_walks_equal_queues_at_odd_sizes(lib_built, w, h, spp):
    sc = scenes.wavelet_grid(3, 24, colors="albedo", light="quad")
    _pair(sc, scenes.orbit_camera(sc), image_w=w, image_h=h, ao_mode=0, pixel_samples=spp, bounces=3)


@pytest.mark.parametrize("bounces", [1, 2, 6])
@pytest.mark.parametrize("wave", [0, 5000])
def test_walks_equal_queues_over_depths_and_waves(lib_built, bounces, wave):
    """One depth runs on one stream, more beside each other's shadow rays; several waves share the buffers."""
    sc = _boxes_scene(27, 5)
    _pair(sc, scenes.orbit_camera(sc), image_w=131, image_h=77, ao_mode=0, ao_samples=2, pixel_samples=3,
          bounces=bounces, wave_samples=wave, max_samples_per_rank=3000)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_walks_equal_queues_for_axis_parallel_rays(lib_built, axis):
    """A camera on a shared plane of the grid looking along an axis: the middle
    row and column of rays have zero direction components and lie in box faces."""
    sc = _boxes_scene(64, 3)
    pos, look = np.full(3, 2.0), np.full(3, 2.0)
    pos[axis] = -6.0
    up = np.eye(3)[(axis + 1) % 3]
    _pair(sc, (pos, look, up), image_w=64, image_h=64, ao_mode=0, pixel_samples=1, bounces=3)


def test_walks_refuse_what_the_lists_cannot_hold(lib_built):
    """40 boxes on one line: a ray along it overlaps more domains than a list holds."""
    base = _boxes_scene(1, 0).domains[0]
    sc = sg.Scene([sg.Domain(base.vertices * 0.5 + np.float32([0, 0, k]), base.faces, base.colors) for k in range(40)], [])
    sc.lights = scenes.make_lights("point", *scenes.scene_box(sc))
    for launches in (0, 4):
        t = sg.Tracer(small_config(image_w=32, image_h=32, bucket_launches=launches))
        t.set_scene(sc)
        t.set_camera((0.2, 0.2, -3.0), (0.2, 0.2, 50.0), (0, 1, 0))
        with pytest.raises(sg.SprayError) as e:
            t.trace()
        assert e.value.code == sg.EOVERFLOW
