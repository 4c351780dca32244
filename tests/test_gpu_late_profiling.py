"""Profiling switched on after a trace: its times are not there, and asking for
them does not make the next trace fail."""
import pytest

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [abi.KERNEL_PLAIN, abi.KERNEL_WAVEFRONT])
def test_times_of_an_unprofiled_trace(tracer_lib, kernel):
    with abi.Tracer(0) as tr:
        tr.upload_scene(soup_scene(3, 500))
        fr = S.frame(S.look_at((0.0, 0.0, 30.0), (0.0, 0.0, 0.0), 40.0), 1.0, 0.4)
        p = abi.Tracer.params(64, 64, spp=2, max_depth=3, kernel=kernel)
        tr.trace(fr, p)
        tr.set_profiling(True)
        assert tr.timings()["total_ms"] == 0.0
        tr.rounds()
        tr.trace(fr, p)
        assert tr.timings()["total_ms"] > 0.0
