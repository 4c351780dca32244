"""The automatic choice on scenes of spheres alone, from 2^22 path bounces: the
wavefront on many unlit ones, the plain kernel (one launch) on few, on lit ones
and on smaller frames; the same bits from both."""
import ctypes

import numpy as np
import pytest

from conftest import fbits

from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lit,height,plain", [
    (512, False, 256, True),
    (513, False, 256, False),
    (513, False, 255, True),   # one row short of 2^22 bounces
    (513, True, 256, True),
])
def test_choice_on_scenes_of_spheres(gpu_tracer, n, lit, height, plain):
    tr, w = gpu_tracer, 1024
    sc = S.Scene(spheres=S.random_spheres(7, n), bvh=S.BVH_MEDIAN, leaf_size=2)
    sc.spheres["mat"]["emissive"] = 0.0
    sc.spheres["r"] *= 0.2
    if lit:
        sc.spheres[0]["mat"] = S.material((1, 1, 1), (30.0, 28.0, 25.0), 0.6, 0.0)
    tr.upload_scene(sc)
    fr = S.frame(S.look_at((0.5, 2.0, 30.0), (0.0, 0.0, 0.0), 45.0), w / height, 0.3)

    def trace(kernel):
        tr.trace(fr, abi.Tracer.params(w, height, spp=4, max_depth=4, rr_start=3, sky=(0.3, 0.2, 0.1), kernel=kernel,
                                       aovs=(abi.AOV_RGBA32F,)))
        t = abi.Timings()  # (with profiling on the choice is another; off, the counts are there, the times not)
        tr.lib.tracer_last_timings(tr.h, ctypes.byref(t))
        return t.launches, fbits(tr.readback(abi.AOV_RGBA32F))

    launches, image = trace(abi.KERNEL_AUTO)
    assert (launches == 1) == plain
    other, want = trace(abi.KERNEL_WAVEFRONT if plain else abi.KERNEL_PLAIN)
    assert (other == 1) != plain
    assert np.array_equal(image, want)
