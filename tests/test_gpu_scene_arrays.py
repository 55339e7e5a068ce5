"""The triangle boxes and records that the device forms from the caller's arrays:
boxes against the host builder's, records against the triangles themselves."""
import numpy as np
import pytest

from rustracer_b200.renderer import GpuScene
from rustracer_b200.scene import Material, SceneBuilder
from tests.test_gpu_bvh_build import _same_bvh

pytestmark = pytest.mark.gpu


def _scene(n, normals, others):
    """n disjoint triangles on a grid, every third of them flat along an axis (a
    padded box), with two materials."""
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.unravel_index(np.arange(n), (side,) * 3), 1).astype(np.float64) - side / 2
    V = np.empty((n, 3, 3))
    for i in range(n):
        t = np.array([[-0.2, -0.2, 0.0], [0.2, -0.2, 0.0], [0.0, 0.2, 0.0]])
        if i % 3:
            t += rng.uniform(-0.05, 0.05, (3, 3))
        V[i] = np.roll(t, i % 2 + (i // 3) % 2, axis=1) + g[i]
    sb = SceneBuilder()
    mats = [sb.add_material(Material.lambertian((0.5, 0.5, 0.5))), sb.add_material(Material.lambertian((0.1, 0.2, 0.3)))]
    h = (n + 1) // 2
    for part, mat in ((V[:h], mats[0]), (V[h:], mats[1])):
        if len(part):
            sb.add_mesh(part.reshape(-1, 3), np.arange(3 * len(part)).reshape(-1, 3), mat,
                        vnormals=rng.normal(size=(3 * len(part), 3)) if normals else None)
    if others:
        sb.add_quad((-9.0, -9.0, -9.0), (18.0, 0, 0), (0, 0, 18.0), mats[0])
        sb.add_sphere((0.0, 9.0, 0.0), 0.7, mats[1])
    return sb, V


@pytest.mark.parametrize("normals", [False, True])
@pytest.mark.parametrize("others", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 1000])
def test_boxes_and_records(n, others, normals):
    sb, V = _scene(n, normals, others)
    if n + others > 1:
        dev = _same_bvh(sb)[1]
    else:                                   # one primitive: nothing to build
        dev = GpuScene(sb)
    # one ray to the centroid of each triangle, from half a cell along its normal
    V = V.astype(np.float32).astype(np.float64)
    c = V.mean(1)
    nr = np.cross(V[:, 1] - V[:, 0], V[:, 2] - V[:, 0])
    nr /= np.linalg.norm(nr, axis=1)[:, None]
    r = np.concatenate([c + 0.3 * nr, -nr, np.full((n, 1), 0.001), np.full((n, 1), np.inf)], 1).astype(np.float32)
    h = dev.trace_closest(r)
    assert np.array_equal(h["prim"], np.arange(n))
    # f32 coordinates up to 6 (half a ulp 2.4e-7) over edges of 0.3: a few 1e-6
    assert np.abs(h["t"] - 0.3).max() < 1e-5
    assert np.abs(h["b1"] - 1 / 3).max() < 1e-4 and np.abs(h["b2"] - 1 / 3).max() < 1e-4
