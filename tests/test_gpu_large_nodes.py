"""The level-by-level split of large BVH nodes (counting sort over 4096-primitive
chunks) against the host builder, at the edges of a chunk and of a warp's run."""
import pytest

from tests.test_gpu_bvh_build import _same_bvh
from tests.test_gpu_small_nodes import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "coincident", "line"])
@pytest.mark.parametrize("n", [511, 513, 4095, 4096, 4097, 8193, 33 * 4096 + 1])
def test_large_nodes_match_the_host_builder(n, kind):
    _same_bvh(_scene(n, kind))
