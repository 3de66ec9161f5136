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
