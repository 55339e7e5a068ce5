"""A triangle whose plane holds the ray: its distance comes out far in front of its
box.  Whether such a hit counts depends on the triangle and the ray, not on which of
two triangles of one node is tested first."""
import numpy as np
import pytest

from oracle import oracle as O
from rustracer_b200.renderer import GpuScene
from rustracer_b200.scene import Material, SceneBuilder
from tests.test_gpu_trace import assert_same_hits

pytestmark = pytest.mark.gpu


def _cases(count, seed):
    """(edge-on triangle, facing triangle, ray): the edge-on one's computed distance
    is the smallest, then the facing one's, then the entry of the edge-on one's box."""
    f = np.float32
    rng = np.random.default_rng(seed)
    n = 100_000
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(f)
    o = rng.uniform(-1, 1, (n, 3)).astype(f)
    w = np.cross(d, rng.normal(size=(n, 3)))
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    nrm = np.cross(d, w)
    c = o + d * rng.uniform(3, 8, (n, 1))
    size, off = 10 ** rng.uniform(-1.5, 0, (n, 1)), 10 ** rng.uniform(-7, -5, (n, 1))
    r = lambda: rng.uniform(-1, 1, (n, 1))
    V = np.stack([(c + size * (r() * d + r() * w + off * r() * nrm)).astype(f) for _ in range(3)])
    cross = lambda a, b: np.stack([a[:, (k + 1) % 3] * b[:, (k + 2) % 3] - a[:, (k + 2) % 3] * b[:, (k + 1) % 3]
                                   for k in range(3)], 1)
    dot = lambda a, b: a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1] + a[:, 2] * b[:, 2]
    e1, e2, s = V[1] - V[0], V[2] - V[0], o - V[0]
    h = cross(d, e2)
    aa = dot(e1, h)
    with np.errstate(all="ignore"):
        inv_a = f(1) / aa
        b1, q = inv_a * dot(s, h), cross(s, e1)
        b2, t = inv_a * dot(d, q), inv_a * dot(e2, q)
        hit = (np.abs(aa) >= 1e-8) & (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b1 + b2 <= 1)
    a, b = (V.min(0) - o) / d, (V.max(0) - o) / d
    near, far = np.minimum(a, b).max(1), np.maximum(a, b).min(1)
    pick = np.where(hit & (t > 0.5) & (t < 0.8 * near) & (near < far))[0][:count]
    for i in pick:
        m = 0.5 * (float(t[i]) + float(near[i]))
        p = o[i] + d[i] * m
        facing = [p + 0.3 * (x * w[i] + y * nrm[i]) for x, y in ((-1, -1), (2, -1), (-1, 2))]
        yield V[:, i], np.array(facing, f), np.concatenate([o[i], d[i], [f(1e-3), f(np.inf)]]).astype(f)


@pytest.mark.parametrize("sign", [1, -1])        # mirrored, the two change places in the node
@pytest.mark.parametrize("fmt", [0, 1, 2])
def test_hits_do_not_depend_on_the_order_in_a_node(sign, fmt):
    found = 0
    for edge, facing, ray in _cases(12, 5):
        sb = SceneBuilder()
        m = sb.add_material(Material.lambertian((0.5, 0.5, 0.5)))
        sb.add_mesh(np.concatenate([edge, facing]) * np.float32(sign), np.arange(6).reshape(-1, 3), m)
        r = ray[None].copy()
        r[:, :6] *= sign
        ref = O.OracleScene(sb).trace_closest(r)
        g = GpuScene(sb)
        g.set_tuning(node_format=fmt)
        assert_same_hits(g.trace_closest(r), ref)
        found += int(ref["prim"][0] == 0)
        g.close()
    assert found >= 10                            # the edge-on triangle is the closest in nearly all
