"""Scenes of triangles, spheres (emitters among them) and planes: the path
kernels trace the triangles over the 8-wide BVH and the rest over the binary
one, with a warp's lanes shading together.  Every form must give the bits of
the canonical traversal (the plain kernel with statistics)."""
import numpy as np
import pytest

from conftest import fbits

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


def _scene(lights, leaf=0, n=700):
    sc = soup_scene(51, n, extent=10.0, sigma=0.6)
    sc.leaf_size = leaf
    sc.spheres = S.random_spheres(9, 9)
    for k in range(lights):
        sc.spheres[k]["mat"] = S.material((1, 1, 1), (30.0, 28.0 - k, 25.0), 0.6, 0.0)
        sc.spheres[k]["P"] = (4.0 * k - 3.0, 12.0, 2.0 * k)
    sc.planes = np.zeros(1, S.PLANE)
    sc.planes[0]["mat"] = S.material((0.8, 0.7, 0.6), roughness=0.4)
    sc.planes[0]["N"], sc.planes[0]["len"] = (0.0, 1.0, 0.0), 12.0
    return sc


def _trace(tr, fr, w, h, kernel, width=0, stats=False, tail=0):
    p = abi.Tracer.params(w, h, spp=3, max_depth=5, rr_start=2, sky=(0.3, 0.2, 0.1), kernel=kernel, bvh_width=width,
                          tail_paths=tail, stats=stats, aovs=(abi.AOV_RGBA8, abi.AOV_RGBA32F, abi.AOV_PRIMARY_HIT))
    tr.trace(fr, p)
    s = tr.stats() if stats else None
    return tr.readback(abi.AOV_RGBA32F), tr.readback(abi.AOV_RGBA8), tr.readback(abi.AOV_PRIMARY_HIT), s


# a leaf of 8 triangles: the scene has no 8-wide BVH and stays binary
@pytest.mark.parametrize("w,h", [(1, 1), (33, 17), (70, 45)])
@pytest.mark.parametrize("lights,leaf", [(0, 0), (1, 0), (3, 0), (2, 8)])
def test_every_form_gives_the_canonical_bits(gpu_tracer, w, h, lights, leaf):
    gpu_tracer.upload_scene(_scene(lights, leaf))
    fr = S.frame(S.look_at((0.0, 3.0, 28.0), (0.0, 0.0, 0.0), 40.0), w / h, 0.37)
    want = _trace(gpu_tracer, fr, w, h, abi.KERNEL_PLAIN, stats=True)
    for kernel, width, tail, stats in ((abi.KERNEL_PLAIN, 0, 0, False), (abi.KERNEL_WAVEFRONT, 0, 0, False),
                                       (abi.KERNEL_WAVEFRONT, 0, 1, True), (abi.KERNEL_WAVEFRONT, 2, 0, True),
                                       (abi.KERNEL_WAVEFRONT, 0, 600, False)):
        got = _trace(gpu_tracer, fr, w, h, kernel, width, stats, tail)
        key = (kernel, width, tail)
        assert np.array_equal(fbits(got[0]), fbits(want[0])), key
        assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2]), key
        if stats:
            for k in ("closest_rays", "shadow_rays", "hits", "plane_tests"):
                assert got[3][k] == want[3][k], (key, k)


def test_adjoint_recomputes_the_linear_image(gpu_tracer):
    """Without a linear image the per-pixel adjoint computes it first: the
    same gradients as with the forward's (sums in another order: 1e-5)."""
    sc = _scene(2)
    gpu_tracer.upload_scene(sc)
    w, h = 37, 21
    fr = S.frame(S.look_at((0.0, 3.0, 28.0), (0.0, 0.0, 0.0), 40.0), w / h, 0.37)
    p = abi.Tracer.params(w, h, spp=2, max_depth=4, rr_start=2, sky=(0.3, 0.2, 0.1), aovs=(abi.AOV_LINEAR,))
    gpu_tracer.trace(fr, p)
    lin = gpu_tracer.readback(abi.AOV_LINEAR)
    dl = np.random.default_rng(3).standard_normal((h, w, 4)).astype(np.float32)
    given = gpu_tracer.trace_adjoint(fr, p, dl, lin, num_materials=len(sc.materials))
    computed = gpu_tracer.trace_adjoint(fr, p, dl, None, num_materials=len(sc.materials))
    for a, b in zip(given, computed):
        scale = float(np.max(np.abs(a)))
        assert scale > 0
        np.testing.assert_allclose(b, a, rtol=1e-5, atol=1e-7 * scale)
