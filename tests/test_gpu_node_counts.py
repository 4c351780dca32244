"""node_fetches counts 32-byte records read: three for a node of the 8-wide
BVH, in the wavefront's rounds as in its finishing kernel.  Over a tree of one
node every ray visits that node once, in either."""
import pytest

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2])
def test_rounds_and_finishing_kernel_count_alike(gpu_tracer, n):
    gpu_tracer.upload_scene(soup_scene(3, n, sigma=3.0))
    w, h = 65, 33
    fr = S.frame(S.look_at((0.0, 0.0, 30.0), (0.0, 0.0, 0.0), 40.0), w / h, 0.4)
    stats = []
    for tail in (1, 0):  # rounds to the end; no round
        gpu_tracer.trace(fr, abi.Tracer.params(w, h, spp=2, max_depth=3, sky=(1, 1, 1), kernel=abi.KERNEL_WAVEFRONT,
                                               tail_paths=tail, stats=True))
        stats.append(gpu_tracer.stats())
    assert stats[0] == stats[1]
    assert stats[0]["node_fetches"] == 3 * stats[0]["closest_rays"]
