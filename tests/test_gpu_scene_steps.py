"""One tracer through a sequence of scenes, views and failed updates: the buffers
and captured launches it keeps between them must never show the last scene."""
import time

import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config

pytestmark = pytest.mark.gpu


def bits(a):
    return a.view(np.uint32)


def _fresh(cfg, scene, cam):
    t = sg.Tracer(cfg)
    t.set_scene(scene)
    t.set_camera(*cam)
    return t.trace()[0]


@pytest.mark.parametrize("shader", ["pt", "ao"])
def test_scenes_one_after_the_other(lib_built, shader):
    cfg = small_config(image_w=53, image_h=41, ao_mode=int(shader == "ao"), ao_samples=3, pixel_samples=2,
                       bounces=1 if shader == "ao" else 3)
    t = sg.Tracer(cfg)
    # domain counts, meshes and lights (shadow rays per hit) grow and shrink
    for grid, mesh, light in ((2, 24, "point"), (3, 20, "point+diffuse"), (1, 32, "quad"), (3, 28, "point+diffuse"),
                              (2, 24, "point")):
        sc = scenes.wavelet_grid(grid, mesh, colors="albedo", light=light)
        cam = scenes.orbit_camera(sc, frame=grid)
        t.set_scene(sc)
        t.set_camera(*cam)
        want = _fresh(cfg, sc, cam)
        for _ in range(3):  # launched directly, captured, replayed
            assert np.array_equal(bits(t.trace()[0]), bits(want))


def test_more_shadow_rays_per_hit_than_the_last_frame(lib_built):
    sc = scenes.wavelet_grid(2, 24, colors="albedo", light="point")
    cfg = small_config(image_w=64, image_h=48, ao_mode=0, pixel_samples=2, bounces=2)
    pos, look, up = scenes.orbit_camera(sc)
    t = sg.Tracer(cfg)
    t.set_scene(sc)
    t.set_camera(pos, look, up)
    first = t.trace()[0]
    view = dict(position=pos, lookat=look, up=up, image_w=64, image_h=48, pixel_samples=2, ao_mode=1, ao_samples=16,
                bounces=1)
    got = t.trace_views([view])[0][0]
    want = _fresh(dict(cfg, ao_mode=1, ao_samples=16, bounces=1), sc, (pos, look, up))
    assert np.array_equal(bits(got), bits(want))
    assert np.array_equal(bits(t.trace()[0]), bits(first))


def test_a_failed_update_leaves_no_scene(lib_built):
    sc = scenes.wavelet_grid(2, 24, colors="albedo", light="point")
    cam = scenes.orbit_camera(sc)
    t = sg.Tracer(small_config(image_w=32, image_h=32))
    t.set_scene(sc)
    t.set_camera(*cam)
    want = t.trace()[0]
    t.trace()
    bad = sg.Scene([sg.Domain(np.zeros((3, 3), np.float32), [[0, 1, 7]])], sc.lights)
    with pytest.raises(sg.SprayError) as e:
        t.set_scene(bad)
    assert e.value.code == sg.EINVAL and "face index" in str(e.value)
    with pytest.raises(sg.SprayError) as e:
        t.trace()
    assert e.value.code == sg.ESTATE
    t.set_scene(sc)
    assert np.array_equal(bits(t.trace()[0]), bits(want))


@pytest.mark.parametrize("order", ["ABA", "ABBA", "BAAB", "BAB", "AABBA"])
@pytest.mark.parametrize("queues", [0, 4])
def test_views_that_differ_in_their_shadow_slots_only(lib_built, order, queues):
    # a captured frame holds the slots per hit: one of A's nine slots (light_shadow) may
    # not be replayed for B's eight, nor the other way round
    sc = scenes.wavelet_grid(2, 24, colors="albedo", light="point")
    pos, look, up = scenes.orbit_camera(sc)
    cfg = small_config(image_w=64, image_h=48, ao_mode=1, ao_samples=8, ao_max_distance=0.5, bucket_launches=queues)
    want = {k: _fresh(dict(cfg, ao_light_shadow=int(k == "A")), sc, (pos, look, up)) for k in "AB"}
    assert not np.array_equal(bits(want["A"]), bits(want["B"]))
    t = sg.Tracer(cfg)
    t.set_scene(sc)
    for k in order:
        view = dict(position=pos, lookat=look, up=up, image_w=64, image_h=48, pixel_samples=1, ao_mode=1, ao_samples=8,
                    ao_max_distance=0.5, ao_light_shadow=int(k == "A"), bounces=1)
        assert np.array_equal(bits(t.trace_views([view])[0][0]), bits(want[k])), k


@pytest.mark.parametrize("bvh_device", [0, 1])
def test_more_vertices_than_the_numbering_holds_are_refused(lib_built, bvh_device):
    # two domains that claim 2^30 vertices each: refused before any is read
    class Claims(sg.Scene):
        def domain_structs(self):
            doms = super().domain_structs()
            for d in doms:
                d.num_vertices = 1 << 30
            return doms

    tri = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
    doms = [sg.Domain(tri + [2 * k, 0, 0], [[0, 1, 2]]) for k in range(2)]
    lights = [sg.Light(0, (0, 0, 9))]
    t = sg.Tracer(small_config(image_w=32, image_h=32, bvh_device=bvh_device))
    with pytest.raises(sg.SprayError) as e:
        t.set_scene(Claims(doms, lights))
    assert e.value.code == sg.EINVAL and "vertex numbering" in str(e.value)
    t.set_scene(sg.Scene(doms, lights))
    t.set_camera((0.5, 0.3, 4), (0.5, 0.3, 0), (0, 1, 0))
    t.trace()


def test_a_large_frames_next_step_keeps_its_buffers(lib_built):
    # the side lists of such a frame (1 GB) are given back while a scene is loaded; the
    # next frame brings back these only (0.6 ms), not every buffer (8 ms, when a new
    # tracer's first frame spent 2 ms on them)
    sc = scenes.wavelet_grid(2, 24, colors="albedo", light="quad")
    cfg = small_config(image_w=1920, image_h=1080, ao_mode=0, ao_samples=1, pixel_samples=16, bounces=3)

    def step(t, scene):
        t.set_scene(scene)
        t.set_camera(*scenes.orbit_camera(scene))
        t0 = time.perf_counter()
        img, st = t.trace()
        return 1e3 * (time.perf_counter() - t0) - st["frame_ms"], img

    step(sg.Tracer(cfg), sc)  # (the library's first frame of this size)
    t = sg.Tracer(cfg)
    first, want = step(t, sc)
    later = [step(t, sc) for _ in range(5)]
    assert all(np.array_equal(bits(img), bits(want)) for _, img in later)
    assert min(ms for ms, _ in later) < 2.0 * first, (first, [ms for ms, _ in later])


@pytest.mark.parametrize("queues", [0, 4])
def test_a_large_frame_after_a_tiny_one(lib_built, queues):
    # the entry arena's size follows the frame, not the first frame ever traced
    sc = scenes.wavelet_grid(4, 24, colors="albedo", light="quad")
    pos, look, up = scenes.orbit_camera(sc)
    cfg = small_config(image_w=16, image_h=16, ao_mode=0, ao_samples=1, pixel_samples=1, bounces=2, bucket_launches=queues)
    t = sg.Tracer(cfg)
    t.set_scene(sc)
    t.set_camera(pos, look, up)
    t.trace()
    view = dict(position=pos, lookat=look, up=up, image_w=512, image_h=512, pixel_samples=4)
    got = t.trace_views([view])[0][0]
    want = _fresh(dict(cfg, image_w=512, image_h=512, pixel_samples=4), sc, (pos, look, up))
    assert np.array_equal(bits(got), bits(want))
