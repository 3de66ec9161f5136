"""set_scene of scenes larger than one upload group, one build batch or the first group
of split levels, against the host builder."""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _sheet(n, at, size=1.0):
    """A wavy sheet of 2 (n - 1)^2 triangles."""
    x, y = np.meshgrid(np.arange(n, dtype=np.float32), np.arange(n, dtype=np.float32), indexing="ij")
    z = np.sin(x * 0.05) * np.cos(y * 0.03) * 12.0
    v = np.stack([x, y, z], -1).reshape(-1, 3) * np.float32(size / n) + np.asarray(at, np.float32)
    i = (np.arange(n - 1)[:, None] * n + np.arange(n - 1)).reshape(-1)
    f = np.concatenate([np.stack([i, i + n, i + 1], 1), np.stack([i + 1, i + n, i + n + 1], 1)]).astype(np.uint32)
    return sg.Domain(v.astype(np.float32), f, np.full(len(v), 0x80a0c0, np.uint32))


def _scene(*domains):
    sc = sg.Scene(list(domains), [])
    sc.lights = scenes.make_lights("point+diffuse", *scenes.scene_box(sc))
    return sc


def _images(sc):
    cfg = small_config(image_w=96, image_h=72, ao_mode=0, ao_samples=2, pixel_samples=2, bounces=2)
    out = []
    for dev in (1, 0):
        t = sg.Tracer(dict(cfg, bvh_device=dev))
        t.set_scene(sc)
        t.set_camera(*scenes.orbit_camera(sc))
        out.append(t.trace()[0])
        t.close()
    assert out[0][..., :3].max() > 0
    assert np.array_equal(bits(out[0]), bits(out[1]))


def _shared_mb():
    """Shared pages of this process: pinned host memory is among them."""
    line = next(l for l in open("/proc/self/status") if l.startswith("RssShmem"))
    return int(line.split()[1]) / 1024


def test_a_domain_larger_than_the_upload_buffer(lib_built):
    # 126 MB of arrays: the buffer that packs domains holds 64 MB at the most
    large, small = _scene(_sheet(1550, (0, 0, 0))), _scene(_sheet(40, (0, 0, 0)), _sheet(60, (1, 0, 0)))
    t = sg.Tracer(small_config(image_w=32, image_h=32))
    t.set_scene(small)
    before = _shared_mb()
    t.set_scene(large)
    assert _shared_mb() - before <= 70.0
    t.close()
    _images(large)


def test_several_upload_groups(lib_built):
    # 40 MB, 126 MB and small domains: groups of their own and a large one between them
    _images(_scene(_sheet(900, (0, 0, 0)), _sheet(900, (1, 0, 0)), _sheet(1550, (2, 0, 0)), _sheet(50, (3, 0, 0)),
                   _sheet(30, (0, 1, 0))))


def test_several_build_batches(lib_built):
    # 17 million triangles: two batches, their nodes joined; out of core every domain
    # keeps its own
    sc = _scene(_sheet(2062, (0, 0, 0)), _sheet(2062, (1, 0, 0)), _sheet(30, (0, 1, 0)))
    cfg = small_config(image_w=96, image_h=72, ao_mode=0, ao_samples=2, pixel_samples=2, bounces=2)
    out = []
    for cache in (-1, 1):
        t = sg.Tracer(dict(cfg, cache_size=cache))
        t.set_scene(sc)
        t.set_camera(*scenes.orbit_camera(sc))
        out.append(t.trace()[0])
        t.close()
    assert out[0][..., :3].max() > 0
    assert np.array_equal(bits(out[0]), bits(out[1]))


def _check_tree(nodes, tris, faces):
    """Every triangle in one leaf, inside its box and all boxes above it."""
    assert np.array_equal(np.sort(tris["v"][:, 0, 3].view(np.uint32)), np.arange(faces))
    v = tris["v"][:, :, :3]
    lo, hi = v.min(1), v.max(1)
    seen = np.zeros(faces, int)

    def walk(k):
        n = nodes[k]
        low, high = np.full(3, np.inf), np.full(3, -np.inf)
        for c in range(4):
            child = int(n["child"][c])
            if child == -2 ** 31:
                continue
            blo, bhi = n["box"][0::2, c], n["box"][1::2, c]
            if child >= 0:
                l, h = walk(child)
            else:
                first, count = (~child) >> 3, ((~child) & 7) + 1
                seen[first:first + count] += 1
                l, h = lo[first:first + count].min(0), hi[first:first + count].max(0)
            assert np.all(blo <= l) and np.all(h <= bhi)
            low, high = np.minimum(low, blo), np.maximum(high, bhi)
        return low, high

    walk(0)
    assert np.all(seen == 1)


@pytest.mark.parametrize("octaves,tail", [(3, 126), (20, 160), (36, 150), (42, 150)])
def test_more_split_levels_than_a_group(lib_built, octaves, tail):
    # a point per octave down to `tail` at one place: every split of a task above 128
    # triangles takes the largest off, 2, 20, 36 and 42 levels (the first group launches
    # 4, then 8 at a time up to 32, then another group)
    s = 2.0 ** -np.minimum(np.arange(octaves + tail), octaves)
    v = np.zeros((octaves + tail, 3, 3), np.float32)
    v[:, :, 0] = s[:, None]
    lopsided = sg.Domain(v.reshape(-1, 3), np.arange(3 * len(v)).reshape(-1, 3))
    sc = _scene(lopsided, _sheet(20, (0.0, -1.0, -0.5)))
    _images(sc)
    t = sg.Tracer(small_config(image_w=32, image_h=32))
    t.set_scene(sc)
    for d, dom in enumerate(sc.domains):
        _check_tree(t.debug(sg.DBG_NODES, d), t.debug(sg.DBG_TRIS, d), len(dom.faces))
