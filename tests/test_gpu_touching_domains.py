"""Surfaces on the boundaries of their domains, where a neighbour's surface may coincide:
the distance of a hit and the entry distance of the domain behind it differ by roundings
only, and leaving that domain out must not change the hit.  Against the oracle, which
looks at every listed domain."""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config

pytestmark = pytest.mark.gpu


def _boxes(n, seed):
    """n closed boxes in the cells of a grid, many faces on common planes."""
    rng = np.random.default_rng(seed)
    corners = np.array([[x, y, z] for z in (0, 1) for y in (0, 1) for x in (0, 1)], np.float32)
    quads = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    faces = np.array([t for a, b, c, d in quads for t in ((a, b, c), (a, c, d))], np.uint32)
    g = int(np.ceil(n ** (1 / 3)))
    doms = []
    for d in range(n):
        size = rng.choice([0.5, 1.0, 1.0, 1.3], 3) * rng.choice([1.0, rng.uniform(0.3, 1.4)])
        v = (np.array([d % g, d // g % g, d // (g * g)]) + corners * size).astype(np.float32)
        doms.append(sg.Domain(v, faces, rng.integers(0, 1 << 24, 8).astype(np.uint32), np.concatenate([v.min(0), v.max(0)])))
    sc = sg.Scene(doms, [])
    sc.lights = scenes.make_lights("point+diffuse", *scenes.scene_box(sc))
    return sc


@pytest.mark.parametrize("n", [8, 27, 64, 100])
@pytest.mark.parametrize("ao", [0, 1])
def test_images_equal_the_oracle(lib_built, oracle_mod, n, ao):
    sc = _boxes(n, n + ao)
    cfg = small_config(image_w=160, image_h=120, ao_mode=ao, ao_samples=3, pixel_samples=2, bounces=1 if ao else 3, list_size=32)
    cam = scenes.orbit_camera(sc, frame=n % 5)
    o = oracle_mod.Oracle(cfg, sc)
    o.set_camera(*cam)
    want = o.render_wavefront()[0].view(np.uint32)
    o.close()
    routes = [dict(), dict(bucket_launches=4), dict(debug_capture=1)]
    routes += [dict(cache_size=max(1, n // 2), schedule_policy=p) for p in (0, 1, 2, 4)]
    wrong = {}
    for kw in routes:
        t = sg.Tracer(dict(cfg, **kw))
        t.set_scene(sc)
        t.set_camera(*cam)
        wrong[str(kw)] = int((t.trace()[0].view(np.uint32) != want).any(-1).sum())
        t.close()
    assert not any(wrong.values()), wrong
