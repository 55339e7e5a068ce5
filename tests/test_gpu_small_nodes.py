"""The warp that finishes a small BVH node against the host builder, at the
sizes where its lanes, its range and its degenerate splits can go wrong."""
import numpy as np
import pytest

from rustracer_b200.scene import Material, SceneBuilder
from tests.test_gpu_bvh_build import _same_bvh

pytestmark = pytest.mark.gpu


def _scene(n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-5, 5, (n, 3))
    if kind == "coincident":                    # no centroid extent: half-span splits
        c[:] = c[0]
    elif kind == "line":                        # one axis with extent, many equal keys
        c[:, 1:] = 0.0
        c[:, 0] = rng.integers(0, 5, n)
    elif kind == "grid":                        # equal costs on several axes and splits
        c = np.stack(np.meshgrid(*[np.arange(6.0)] * 3), -1).reshape(-1, 3)[rng.permutation(216)[:n] % 216]
    shape = np.array([[-0.2, -0.2, 0.0], [0.2, -0.2, 0.1], [0.0, 0.2, -0.1]])
    sb = SceneBuilder()
    V = (c[:, None, :] + shape[None]).reshape(-1, 3)
    sb.add_mesh(V, np.arange(3 * n).reshape(-1, 3), sb.add_material(Material.lambertian((0.5, 0.5, 0.5))))
    return sb


@pytest.mark.parametrize("kind", ["random", "coincident", "line", "grid"])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 191, 192, 193, 400])
def test_small_nodes_match_the_host_builder(n, kind):
    if kind == "grid" and n > 216:
        pytest.skip("the grid has 216 points")
    _same_bvh(_scene(n, kind))
