"""Linear scans (no BVH) in the wavefront and its adjoint: lanes that go their
own ways in the finishing kernels, scans above and below the length from which
shade starts a pixel's next sample at once, the hit log's two passes.  Images
have the bits of the canonical traversal; gradients are those of the adjoint
without a log."""
import numpy as np
import pytest

from conftest import fbits

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


def _scene(kind):
    if kind.startswith("ref"):
        sc = S.reference_scene()
        if kind == "ref unlit":
            sc.spheres["mat"]["emissive"] = 0.0
        return sc, S.reference_frame(0.3), abi.TIES_REFERENCE
    sc = soup_scene(21, 60, sigma=2.0)  # more primitives than a short scan's
    sc.bvh = S.BVH_NONE
    if kind == "lit":
        sc.spheres = S.random_spheres(3, 3)
        sc.spheres["mat"]["emissive"] = 0.0
        sc.spheres[0]["mat"] = S.material((1, 1, 1), (30.0, 28.0, 25.0), 0.6, 0.0)
        sc.spheres[0]["P"] = (0.0, 14.0, 2.0)
    return sc, S.frame(S.look_at((0.5, 2.0, 30.0), (0.0, 0.0, 0.0), 45.0), 1.5, 0.3), abi.TIES_STRICT


@pytest.mark.parametrize("kind", ["ref", "ref unlit", "tris", "lit"])
@pytest.mark.parametrize("w,h", [(1, 1), (67, 45)])
def test_scans(gpu_tracer, kind, w, h):
    tr = gpu_tracer
    sc, fr, tie = _scene(kind)
    tr.upload_scene(sc)

    def params(kernel, tail=0, stats=False, spp=3):
        return abi.Tracer.params(w, h, spp=spp, max_depth=4, rr_start=2, sky=(0.3, 0.2, 0.1), tie_mode=tie,
                                 kernel=kernel, tail_paths=tail, stats=stats, aovs=(abi.AOV_RGBA32F, abi.AOV_LINEAR))

    for spp in (1, 3):
        tr.trace(fr, params(abi.KERNEL_PLAIN, stats=True, spp=spp))
        want = fbits(tr.readback(abi.AOV_RGBA32F))
        assert w == 1 or len(np.unique(want[:, 1:].reshape(-1, 4), axis=0)) > 8
        for tail in (0, 1, 900):  # no round; rounds to the end; a hand-over between
            for stats in (False, True):
                tr.trace(fr, params(abi.KERNEL_WAVEFRONT, tail, stats, spp))
                assert np.array_equal(fbits(tr.readback(abi.AOV_RGBA32F)), want), (spp, tail, stats)
    lin = tr.readback(abi.AOV_LINEAR)
    dl = np.random.default_rng(2).standard_normal((h, w, 4)).astype(np.float32)
    n_mat = max(1, len(sc.materials))
    plain = tr.trace_adjoint(fr, params(abi.KERNEL_PLAIN), dl, lin, num_materials=n_mat)
    for log in (0, 1 << 26):
        tr.set_adjoint_hit_log(log)
        try:
            for tail in (0, 1, 900):
                got = tr.trace_adjoint(fr, params(abi.KERNEL_WAVEFRONT, tail), dl, lin, num_materials=n_mat)
                for a, b in zip(got, plain):  # FP64 sums in another order
                    np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-7 * max(1e-30, float(np.max(np.abs(b)))))
        finally:
            tr.set_adjoint_hit_log(0)
