"""Closest hits over quantised nodes, whose lanes test their pending leaves while
others visit nodes: the same hits as over 4-wide nodes, at ray counts around a warp
and a refill, and with several overlapping leaves per node."""
import numpy as np
import pytest

from rustracer_b200.renderer import GpuScene
from rustracer_b200.scene import Material, SceneBuilder

pytestmark = pytest.mark.gpu


def _scene(kind):
    rng = np.random.default_rng(3)
    n = {"pair": 2, "node": 8, "stack": 64, "soup": 4000}[kind]
    c = rng.uniform(-2, 2, (n, 3)) * ((0.02, 0.02, 1.0) if kind == "stack" else (1.0, 1.0, 1.0))
    V = c[:, None, :] + rng.uniform(-0.6, 0.6, (n, 3, 3)) * (1.0 if kind != "soup" else 0.3)
    sb = SceneBuilder()
    sb.add_mesh(V.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3), sb.add_material(Material.lambertian((0.5, 0.5, 0.5))))
    return GpuScene(sb)


@pytest.mark.parametrize("kind", ["pair", "node", "stack", "soup"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 5000])
def test_same_hits_as_over_4_wide_nodes(kind, n):
    g = _scene(kind)
    rng = np.random.default_rng(n)
    o = rng.uniform(-3, 3, (n, 3))
    d = rng.uniform(-1, 1, (n, 3)) - o if kind != "soup" else rng.normal(size=(n, 3))
    r = np.concatenate([o, d, np.full((n, 1), 0.001), np.full((n, 1), np.inf)], 1).astype(np.float32)
    r[::7, 7] = 0.5                              # short rays end at once
    r[5::11, 3] = np.nan                         # and NaN rays before their first visit
    g.set_tuning(node_format=2)
    wide4 = g.trace_closest(r)
    g.set_tuning(node_format=1)
    split = g.trace_closest(r)
    for k in wide4.dtype.names:
        assert np.array_equal(wide4[k].view(np.uint32), split[k].view(np.uint32)), k
