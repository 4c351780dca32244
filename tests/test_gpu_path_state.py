"""Device memory of the wavefront's path state in a context's first trace: the
primary hits (16 bytes a pixel) are held only where later samples read them."""
import pytest
import torch

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu

SIDE = 2048


def _held(spp, stats):
    with abi.Tracer(0) as tr:
        tr.upload_scene(soup_scene(3, 50))
        fr = S.frame(S.look_at((0.0, 0.0, 30.0), (0.0, 0.0, 0.0), 40.0), 1.0, 0.4)
        tr.synchronize()
        before = torch.cuda.mem_get_info()[0]
        tr.trace(fr, abi.Tracer.params(SIDE, SIDE, spp=spp, max_depth=2, kernel=abi.KERNEL_WAVEFRONT, stats=stats))
        tr.synchronize()
        return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("spp,stats", [(1, False), (2, True)])
def test_no_room_for_hits_that_nothing_reads(tracer_lib, spp, stats):
    _held(2, False)  # the kernels' own memory, taken as they are first launched
    _held(spp, stats)
    saved = _held(2, False) - _held(spp, stats)
    assert abs(saved - 16 * SIDE * SIDE) <= 4 << 20  # allocations are rounded up to 2 MB
