"""A photon map that does not fit into the device's memory is refused, and the scene
stays usable: a smaller map is built and read afterwards."""
import numpy as np
import pytest
import torch

from rustracer_b200 import configs
from rustracer_b200.renderer import GpuScene, RtError

pytestmark = pytest.mark.gpu


def _map(n, seed):
    rng = np.random.default_rng(seed)
    nor = np.tile(np.float32([0, 1, 0]), (n, 1))
    return rng.uniform(0, 1, (n, 3)).astype(np.float32), rng.uniform(0, 1, (n, 3)).astype(np.float32), nor


# free memory: a part of the map's arrays fits, 9 of 16 B and their keys a photon
@pytest.mark.parametrize("spare_mb", [96, 288, 480])
def test_a_map_too_large_leaves_the_scene_usable(spare_mb):
    sb, _ = configs.box_scene(width=16, height=16)
    g = GpuScene(sb)
    q = np.concatenate([_map(200, 1)[0], np.tile(np.float32([0, 1, 0]), (200, 1))], 1)
    pos, power, nor = _map(900, 2)
    g.photon_set(pos, power, nor, radius=0.2, knn_k=8)
    ref = g.photon_gather(q)
    assert (ref > 0).any()
    large = _map(4_000_000, 3)                       # 64 MB an array
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (spare_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(RtError):
            g.photon_set(*large, radius=0.2, knn_k=8)
        g.photon_set(pos[:500], power[:500], nor[:500], radius=0.2, knn_k=8)
        few = g.photon_gather(q)
    finally:
        del fill
        torch.cuda.empty_cache()
    h = GpuScene(sb)
    h.photon_set(pos[:500], power[:500], nor[:500], radius=0.2, knn_k=8)
    assert np.array_equal(few.view(np.uint32), h.photon_gather(q).view(np.uint32))
    g.photon_set(*large, radius=0.2, knn_k=8)        # and the large one once there is room
    g.photon_set(pos, power, nor, radius=0.2, knn_k=8)
    assert np.array_equal(g.photon_gather(q).view(np.uint32), ref.view(np.uint32))
