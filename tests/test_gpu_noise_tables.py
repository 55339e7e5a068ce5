"""The media kernels' shared noise tables: the first noise medium of a scene
reads them, later ones the global tables, so the same media in the other order
must give the same image bit for bit."""
import numpy as np
import pytest

from rustracer_b200 import configs
from rustracer_b200.renderer import GpuScene, pass_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(3, 2, 1), (37, 29, 2), (96, 64, 8)])
def test_noise_media_in_either_order_render_identically(w, h, spp):
    def scene(order):
        sb, st = configs.box_scene(w, h, spp, 24, 4, 5)
        sb.spheres.clear()
        media = [dict(density=5.0, color=(0.9, 0.8, 0.7), g=0.3, noise_scale=4.0, threshold=0.05, seed=11,
                      p_min=(0.0, 0.0, 0.0), p_max=(1.0, 0.5, 1.0)),
                 dict(density=8.0, color=(0.7, 0.8, 0.9), g=-0.2, noise_scale=9.0, threshold=0.0, seed=12,
                      p_min=(0.1, 0.3, 0.1), p_max=(0.9, 0.9, 0.8))]
        for k in order:
            sb.add_medium("noise", "box", **media[k])
        return GpuScene(sb), st
    p = pass_params(w, h, 0, spp, max_depth=24, hero=4, seed=9)
    (a, st), (b, _) = scene((0, 1)), scene((1, 0))
    x, y = a.render_pass(st["camera"], p), b.render_pass(st["camera"], p)
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32)) and (w * h < 100 or x.max() > 0)
