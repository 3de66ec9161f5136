"""The image sums of the GPU against the oracle at samples per pixel whose
reciprocal is and is not a power of two (the sums take different paths)."""
import numpy as np
import pytest

import spray_gb300 as sg
from spray_gb300 import scenes
from conftest import small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 2, 3, 5, 6, 7, 16, 33])
@pytest.mark.parametrize("ao", [0, 1])
def test_image_sums_equal_the_oracle(lib_built, oracle_mod, spp, ao):
    sc = scenes.wavelet_grid(2, 24, colors="albedo", light="point+diffuse")
    cfg = small_config(image_w=37, image_h=29, ao_mode=ao, ao_samples=3, pixel_samples=spp, bounces=1 if ao else 3)
    cam = scenes.orbit_camera(sc)
    t = sg.Tracer(cfg)
    t.set_scene(sc)
    t.set_camera(*cam)
    img, _ = t.trace()
    o = oracle_mod.Oracle(cfg, sc)
    o.set_camera(*cam)
    want, _ = o.render_wavefront()
    assert np.array_equal(img.view(np.uint32), want.view(np.uint32))
