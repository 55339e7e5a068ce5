"""The packed nodes (children in octant slots, one header, leaf references as
hit records) and the warp's convex test against the oracle, bit for bit, where
they can go wrong: one node, full and part-filled nodes, the sizes where the
launch changes layout, rays on the fast and the general slab path, plane
counts around a warp's 32 lanes."""
import numpy as np
import pytest

from oracle import oracle as O
from rustracer_b200.renderer import GpuScene
from rustracer_b200.scene import Material, SceneBuilder
from tests.test_gpu_trace import assert_same_hits

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    sb = SceneBuilder()
    m = sb.add_material(Material.lambertian((0.5, 0.5, 0.5)))
    c = rng.uniform(-2, 2, (n, 1, 3))
    sb.add_mesh((c + rng.normal(0, 2.0 / n ** (1 / 3), (n, 3, 3))).reshape(-1, 3), np.arange(3 * n).reshape(-1, 3), m)
    return sb


def _hard_rays(seed, n=6000):
    """Random rays, and the ones the general slab path takes: zero and denormal
    direction components, negative t_min, extreme magnitudes, NaN; origins on
    axis planes, short and empty intervals."""
    rng = np.random.default_rng(seed)
    o, d = rng.uniform(-3, 3, (n, 3)), rng.normal(size=(n, 3))
    t0, t1 = np.full(n, 0.001), np.full(n, np.inf)
    k = n // 12
    d[0:k, 0] = 0.0
    d[k:2 * k, 1:] = 0.0
    d[2 * k:3 * k, 2] = 1e-42
    d[3 * k:4 * k] *= 1e-20
    d[4 * k:5 * k] *= 1e20
    o[5 * k:6 * k, 1] = 0.0
    t0[6 * k:7 * k] = -1.0
    t1[7 * k:8 * k] = rng.uniform(0, 3, k)
    t0[8 * k:9 * k], t1[8 * k:9 * k] = 2.0, 1.0
    o[9 * k:10 * k] *= 1e4
    d[9 * k:10 * k] = -o[9 * k:10 * k]
    o[10 * k] = np.nan
    d[10 * k + 1] = -0.0
    return np.concatenate([o, d, t0[:, None], t1[:, None]], 1).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 65, 1200, 3000])
def test_packed_nodes_give_the_oracle_hits(n):
    sb = _soup(n, n)
    g, o = GpuScene(sb), O.OracleScene(sb)
    r = _hard_rays(n)
    ref, occ = o.trace_closest(r), o.trace_any(r)
    for fmt in (0, 1, 2) if n >= 2 else (0, 1):      # one primitive: its node is the host's, which has no 4-wide form
        g.set_tuning(node_format=fmt)
        assert_same_hits(g.trace_closest(r), ref)
        assert np.array_equal(g.trace_any(r), occ), fmt
    g.set_tuning(stack_ring=1)                       # every pending group goes through the spill columns
    assert_same_hits(g.trace_closest(r), ref)


@pytest.mark.parametrize("planes", [4, 31, 32, 33, 64, 97, 700])
def test_warp_convex_test_gives_the_oracle_hits(planes):
    """Solids of `planes` half-spaces (a box or a tetrahedron cut by random
    planes), nested and overlapping, so one visit meets several of them."""
    rng = np.random.default_rng(planes)
    sb = SceneBuilder()
    m = sb.add_material(Material.dielectric(1.5))
    for k in range(5):
        base = np.array([[1, 1, 1], [-1, -1, 1], [-1, 1, -1], [1, -1, -1]], float) / np.sqrt(3)
        extra = rng.normal(size=(planes - 4, 3))
        nv = np.concatenate([base, extra / np.maximum(np.linalg.norm(extra, axis=1, keepdims=True), 1e-9)])
        pl = np.concatenate([nv, np.full((planes, 1), 0.5)], 1).astype(np.float32)
        sb.add_convex(pl, m, (-1.6, -1.6, -1.6), (1.6, 1.6, 1.6), translate=tuple(rng.uniform(-0.6, 0.6, 3)))
    sb.add_quad((-3, -1.2, -3), (6, 0, 0), (0, 0, 6), sb.add_material(Material.lambertian((0.5, 0.5, 0.5))))
    g, o = GpuScene(sb), O.OracleScene(sb)
    r = _hard_rays(planes, 3000)
    ref, occ = o.trace_closest(r), o.trace_any(r)
    for fmt in (0, 1, 2):
        g.set_tuning(node_format=fmt)
        assert_same_hits(g.trace_closest(r), ref)
        assert np.array_equal(g.trace_any(r), occ), fmt
    # intervals that end exactly at the crossing
    hit = ref["prim"] >= 0
    r2 = r[hit].copy()
    r2[:, 7] = ref["t"][hit]
    g.set_tuning()
    assert_same_hits(g.trace_closest(r2), o.trace_closest(r2))
