"""The render path's caustic gather (a lane or a warp per request over the fine
cell grid) against the ray-level gather of the same map: on a bare diffuse
plane one bounce of a pixel is albedo × the irradiance at its hit point."""
import numpy as np
import pytest

from rustracer_b200.renderer import GpuScene, pass_params
from rustracer_b200.scene import Material, SceneBuilder, make_camera

pytestmark = pytest.mark.gpu


def _map(n, kind, seed, off):
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 3))
    if kind == "spread":
        pos[:, [0, 2]] = rng.uniform(-2, 2, (n, 2))
    elif kind == "cluster":                      # most requests see none, a few thousands
        pos[:, [0, 2]] = rng.normal(0, 0.05, (n, 2))
    else:                                        # photons and cell faces at the same coordinates
        pos[:, [0, 2]] = rng.integers(-8, 9, (n, 2)) * 0.25
    pos[:, 1] = rng.choice([0.0, 1e-6, -1e-6], n)
    nor = np.tile([0.0, 1.0, 0.0], (n, 1))
    nor[rng.random(n) < 0.2] *= -1.0             # facing away: not counted
    return pos + off, rng.uniform(0.0, 1.0, (n, 3)), nor


@pytest.mark.parametrize("size", [(24, 16), (192, 128)])       # all warps' requests; lanes' and warps'
@pytest.mark.parametrize("n,kind,radius,k,off", [
    (1, "spread", 0.5, 0, 0.0), (50, "spread", 0.5, 8, 0.0), (3000, "spread", 0.25, 0, 0.0),
    (3000, "spread", 0.25, 16, 0.0), (6000, "cluster", 0.3, 0, 0.0), (6000, "cluster", 0.3, 64, 0.0),
    (900, "cluster", 0.1, 64, 0.0), (4000, "lattice", 0.25, 0, 0.0), (4000, "lattice", 0.25, 32, 0.0),
    (3000, "spread", 0.02, 0, 500.0), (3000, "spread", 0.02, 4, 500.0), (500, "spread", 40.0, 0, 0.0)])
def test_render_gather_matches_the_query_gather(size, n, kind, radius, k, off):
    W, H = size
    albedo = np.array([0.7, 0.5, 0.3], np.float32)
    sb = SceneBuilder()
    sb.set_solid((0.0, 0.0, 0.0))
    sb.add_quad((off - 3, off, off - 3), (0, 0, 6), (6, 0, 0), sb.add_material(Material.lambertian(tuple(albedo))))
    sb.add_sphere((off, off + 9.0, off), 0.1, sb.add_material(Material.lambertian((0.5, 0.5, 0.5))))
    g = GpuScene(sb)
    cam = make_camera((off, off + 4.0, off + 0.5), (off, off, off), vfov=50.0, aspect=W / H)
    pos, power, nor = _map(n, kind, n + k, off)
    g.photon_set(pos, power, nor, radius=radius, knn_k=k)
    p = pass_params(W, H, 0, 1, max_depth=1, hero=1, seed=5, strata=1)
    img = g.render_pass(cam, p)[0].reshape(-1, 3)
    rays = g.capture_rays(cam, p, 0, W * H)
    hit = g.trace_closest(rays)
    floor = hit["prim"] == 0
    assert floor.sum() > 0.5 * W * H
    o, d, t = rays[:, :3], rays[:, 3:6], hit["t"][:, None]
    q = (o + (t * d).astype(np.float32)).astype(np.float32)
    irr = g.photon_gather(np.concatenate([q, np.tile(np.float32([0, 1, 0]), (len(q), 1))], 1))
    want = np.where(floor[:, None], irr * albedo, 0.0)
    # sums of at most n positive terms in two orders: each within (n + 8)·2^-24 of the exact sum
    tol = 2.0 * (n + 8) * 2.0 ** -24
    # the captured rays are in generation order, the image in pixel order: compare as sorted values
    a, b = np.sort(img, axis=0), np.sort(want.astype(np.float32), axis=0)
    assert np.allclose(a, b, rtol=tol, atol=0.0), np.abs(a - b).max()
    if kind == "spread" and radius >= 0.25 and n > 1:
        assert (b > 0).any()
