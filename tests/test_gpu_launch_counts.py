"""last_stats() counts every launch of an iteration that media add."""
import pytest

from rustracer_b200 import configs
from rustracer_b200.renderer import GpuScene, pass_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_media_add_three_launches_an_iteration(graph):
    """Scatter distances, the shading of medium events and the shadow rays'
    transmittance; one bounce is one iteration."""
    n = []
    for media in (True, False):
        sb, st = configs.media_box_scene(width=32, height=32)
        if not media:
            sb.media.clear()
        g = GpuScene(sb)
        g.set_tuning(graph=graph)
        g.render_pass(st["camera"], pass_params(32, 32, 0, 1, 1, 1, 1, 1.0, 3))
        n.append(g.last_stats()["launches"])
    assert n[0] - n[1] == 3
