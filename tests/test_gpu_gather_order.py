"""The caustic lookup of a request is the same sum, bit for bit, however many
other requests are in flight: few (each by a warp) or many (most by a lane)."""
import numpy as np
import pytest

from rustracer_b200.renderer import GpuScene, pass_params
from rustracer_b200.scene import Material, SceneBuilder, make_camera

pytestmark = pytest.mark.gpu

CAM = dict(eye=(0.0, 4.0, 0.5), at=(0.0, 0.0, 0.0), vfov=50.0)


def _scene(k):
    """A diffuse floor under a map of 20,000 photons: about 110 in the cells a
    request meets, 40 in its radius."""
    rng = np.random.default_rng(3)
    pos = np.zeros((20000, 3))
    pos[:, [0, 2]] = rng.uniform(-2, 2, (20000, 2))
    nor = np.tile([0.0, 1.0, 0.0], (20000, 1))
    sb = SceneBuilder()
    sb.set_solid((0.0, 0.0, 0.0))
    sb.add_quad((-3, 0, -3), (0, 0, 6), (6, 0, 0), sb.add_material(Material.lambertian((0.7, 0.5, 0.3))))
    sb.add_sphere((0.4, 0.5, 0.0), 0.5, sb.add_material(Material.lambertian((0.5, 0.5, 0.5))))
    g = GpuScene(sb)
    g.photon_set(pos, rng.uniform(0.0, 1.0, (20000, 3)), nor, radius=0.1, knn_k=k)
    return g


def _cam(w, h):
    return make_camera(CAM["eye"], CAM["at"], vfov=CAM["vfov"], aspect=w / h)


@pytest.mark.parametrize("k", [0, 24, 4096])
def test_samples_per_pass(k):
    g, w, h = _scene(k), 160, 112
    few = g.render_pass(_cam(w, h), pass_params(w, h, 0, 1, 1, 3, 1, 1.0, 5))
    many = g.render_pass(_cam(w, h), pass_params(w, h, 0, 16, 1, 3, 1, 1.0, 5))
    assert (few > 0).mean() > 0.5
    assert np.array_equal(few[0].view(np.uint32), many[0].view(np.uint32))


@pytest.mark.parametrize("k", [0, 24, 4096])
def test_packed_batch(k):
    g = _scene(k)
    reqs = [dict(cam=_cam(120 + 8 * j, 96), width=120 + 8 * j, height=96, spp=1, seed=3 + j) for j in range(8)]
    res, _ = g.render_batch(reqs, pass_params(8, 8, 0, 1, 1, 3, 1, 1.0, 0))
    for r, q in zip(res, reqs):
        alone = g.render_accumulate(q["cam"], pass_params(q["width"], q["height"], 0, 1, 1, 3, 1, 1.0, q["seed"]))
        assert np.array_equal(np.asarray(r[0]).view(np.uint32).ravel(), alone[0].view(np.uint32).ravel())
