"""The node layouts by name: each can be chosen on a scene of any size, the library's
own choice has a value of its own, and all give the oracle's hits and one image."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from rustracer_b200 import abi, configs
from rustracer_b200.renderer import GpuScene, RtError, lib, pass_params
from rustracer_b200.scene import Material, SceneBuilder, make_camera
from tests.test_gpu_packed_nodes import _hard_rays, _soup
from tests.test_gpu_trace import assert_same_hits

pytestmark = pytest.mark.gpu


def _set_layout(g):
    t = abi.RtTuning()
    assert lib().rt_get_tuning(g.h, C.byref(t)) == 0
    return t.node_format


def test_the_layout_that_was_set_is_reported():
    g = GpuScene(_soup(3000, 3))
    assert _set_layout(g) == abi.RT_NODES_AUTO and g.get_tuning()["node_auto"]
    for fmt in (abi.RT_NODES_FULL, abi.RT_NODES_QUANTISED, abi.RT_NODES_WIDE4):
        g.set_tuning(node_format=fmt)
        assert _set_layout(g) == fmt
        g.set_tuning(**g.get_tuning())
        assert _set_layout(g) == fmt and not g.get_tuning()["node_auto"]
    g.set_tuning(max_paths=1 << 20)
    assert _set_layout(g) == abi.RT_NODES_AUTO
    g.set_tuning(**g.get_tuning())
    assert _set_layout(g) == abi.RT_NODES_AUTO
    with pytest.raises(RtError):
        g.set_tuning(node_format=4)


def _solids_in_a_soup():
    """Convex solids among enough triangles for several hundred nodes."""
    sb = _soup(4000, 11)
    m = sb.add_material(Material.lambertian((0.6, 0.4, 0.3)))
    rng = np.random.default_rng(4)
    for _ in range(6):
        nv = rng.normal(size=(40, 3))
        nv = np.concatenate([nv / np.linalg.norm(nv, axis=1, keepdims=True), np.eye(3), -np.eye(3)])
        pl = np.concatenate([nv, np.full((len(nv), 1), 0.3)], 1).astype(np.float32)
        sb.add_convex(pl, m, (-0.4, -0.4, -0.4), (0.4, 0.4, 0.4), translate=tuple(rng.uniform(-1.5, 1.5, 3)))
    return sb


SCENES = {"triangles": lambda: _soup(20000, 7), "solids": _solids_in_a_soup}


@pytest.mark.parametrize("ring", [0, 1])
@pytest.mark.parametrize("kind", sorted(SCENES))
def test_every_layout_of_a_large_scene_gives_the_oracle_hits(kind, ring):
    sb = SCENES[kind]()
    g, o = GpuScene(sb), O.OracleScene(sb)
    assert g.bvh_stats()["nodes"] > 256
    r = _hard_rays(17)
    ref, occ = o.trace_closest(r), o.trace_any(r)
    for fmt in (abi.RT_NODES_FULL, abi.RT_NODES_QUANTISED, abi.RT_NODES_WIDE4, abi.RT_NODES_AUTO):
        g.set_tuning(node_format=fmt, stack_ring=ring)
        assert_same_hits(g.trace_closest(r), ref)
        assert np.array_equal(g.trace_any(r), occ), fmt


@pytest.mark.parametrize("kind", sorted(SCENES))
def test_every_layout_renders_one_image(kind):
    """Also with a one-entry ring, where the extension and the shadow rays, which run
    at the same time, both keep their stacks in global memory, and as one graph."""
    sb = SCENES[kind]()
    sb.set_solid((0.6, 0.7, 0.9))
    sb.add_light_quad((-1, 4, -1), (2, 0, 0), (0, 0, 2), sb.add_material(Material.diffuse_light((9, 9, 9))))
    g = GpuScene(sb)
    cam = make_camera((0.0, 1.0, 6.0), (0.0, 0.0, 0.0), vfov=45.0, aspect=4 / 3)
    p = pass_params(160, 120, 0, 8, 2, 6, 4, 1.0, 11)
    ref = g.render_pass(cam, p).view(np.uint32)
    for fmt in (abi.RT_NODES_FULL, abi.RT_NODES_QUANTISED, abi.RT_NODES_WIDE4, abi.RT_NODES_AUTO):
        for t in (dict(), dict(stack_ring=1), dict(stack_ring=1, graph=1)):
            g.set_tuning(node_format=fmt, **t)
            assert np.array_equal(g.render_pass(cam, p).view(np.uint32), ref), (fmt, t)
