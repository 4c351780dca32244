"""A pixel's primary hit and its later samples in the wavefront: kept and gone
on from in shade, kept for the finishing kernel only (lit scenes without
triangles), not kept (one sample).  Every form gives the bits of the canonical
traversal (the plain kernel with statistics), in a frame and in a batch."""
import numpy as np
import pytest

from conftest import fbits

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


def _scene(kind):
    sc = soup_scene(5, 300, sigma=0.8) if "mixed" in kind else S.Scene(bvh=S.BVH_MEDIAN, leaf_size=2)
    sc.spheres = S.random_spheres(9, 30)
    sc.spheres["mat"]["emissive"] = 0.0
    if "lit" in kind:
        for k in range(2):
            sc.spheres[k]["mat"] = S.material((1, 1, 1), (30.0, 28.0, 25.0), 0.6, 0.0)
            sc.spheres[k]["P"] = (6.0 * k - 3.0, 12.0, 2.0)
    return sc


@pytest.mark.parametrize("spp", [1, 3])
@pytest.mark.parametrize("kind", ["spheres", "lit spheres", "mixed", "lit mixed"])
def test_kept_hits_give_the_canonical_bits(gpu_tracer, kind, spp):
    w, h = 67, 45
    sc = _scene(kind)
    fr = S.frame(S.look_at((0.5, 2.0, 30.0), (0.0, 0.0, 0.0), 45.0), w / h, 0.3)

    def params(kernel, tail=0, stats=False):
        return abi.Tracer.params(w, h, spp=spp, max_depth=4, rr_start=2, sky=(0.3, 0.2, 0.1), kernel=kernel,
                                 tail_paths=tail, stats=stats, aovs=(abi.AOV_RGBA8, abi.AOV_RGBA32F))

    gpu_tracer.upload_scene(sc)
    gpu_tracer.trace(fr, params(abi.KERNEL_PLAIN, stats=True))
    want = gpu_tracer.readback(abi.AOV_RGBA32F)
    assert len(np.unique(want[:, 1:].reshape(-1, 4), axis=0)) > 8
    for tail in (0, 1, 900):  # no round; rounds to the end; a hand-over between
        gpu_tracer.trace(fr, params(abi.KERNEL_WAVEFRONT, tail))
        assert np.array_equal(fbits(gpu_tracer.readback(abi.AOV_RGBA32F)), fbits(want)), tail
    gpu_tracer.upload_scenes([sc, sc])
    for tail in (1, 900):
        for _ in range(2):  # a launched batch, a replay of its graph
            gpu_tracer.trace_batched([fr, fr], [params(abi.KERNEL_WAVEFRONT, tail)] * 2, use_graph=True)
            got = [gpu_tracer.readback_scene(i, abi.AOV_RGBA32F).copy() for i in range(2)]
            assert all(np.array_equal(fbits(g), fbits(want)) for g in got), tail
