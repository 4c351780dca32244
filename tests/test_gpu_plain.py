"""The plain kernel's forms -- with and without next-event code, triangles-only
over the 8-wide BVH, linear scans -- in both register budgets (frames up to
and above 512 pixels an SM): each must give the bits of the canonical traversal
(the plain kernel with statistics), as must the automatic choice of a kernel."""
import numpy as np
import pytest

from conftest import fbits

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu


def _scene(kind):
    lights = 2 if kind.startswith("lit") else 0
    if kind.endswith("linear"):
        sc = S.reference_scene()
        if not lights:
            sc.spheres["mat"]["emissive"] = 0.0
        return sc
    tris = 0 if kind == "spheres" else 3000 if kind != "one" else 1
    sc = soup_scene(61, tris, extent=10.0, sigma=0.4) if tris else S.Scene(bvh=S.BVH_SAH, leaf_size=2)
    sc.leaf_size = 8 if kind == "binary" else sc.leaf_size  # no 8-wide BVH: too many triangles a leaf
    if kind in ("mixed", "lit", "spheres"):
        sc.spheres = S.random_spheres(40, 9)
        sc.spheres["mat"]["emissive"] = 0.0
        for k in range(lights):
            sc.spheres[k]["mat"] = S.material((1, 1, 1), (30.0, 28.0 - k, 25.0), 0.6, 0.0)
            sc.spheres[k]["P"] = (4.0 * k - 3.0, 12.0, 2.0 * k)
    if kind != "one":
        sc.planes = np.zeros(1, S.PLANE)
        sc.planes[0]["mat"] = S.material((0.8, 0.7, 0.6), roughness=0.4)
        sc.planes[0]["N"], sc.planes[0]["len"] = (0.0, 1.0, 0.0), 12.0
    return sc


@pytest.mark.parametrize("w,h", [(1, 1), (67, 45), (401, 307)])
@pytest.mark.parametrize("kind", ["triangles", "one", "binary", "mixed", "lit", "spheres", "linear", "lit linear"])
def test_plain_forms_give_the_canonical_bits(gpu_tracer, kind, w, h):
    tr = gpu_tracer
    sc = _scene(kind)
    tr.upload_scene(sc)
    fr = (S.reference_frame(0.3) if kind.endswith("linear")
          else S.frame(S.look_at((0.5, 2.0, 30.0), (0.0, 0.0, 0.0), 45.0), w / h, 0.3))
    aovs = (abi.AOV_RGBA8, abi.AOV_RGBA32F, abi.AOV_PRIMARY_HIT)

    def trace(kernel, stats):
        tr.trace(fr, abi.Tracer.params(w, h, spp=2, max_depth=5, rr_start=2, sky=(0.3, 0.2, 0.1), kernel=kernel,
                                       stats=stats, aovs=aovs))
        return [tr.readback(a) for a in aovs]

    want = trace(abi.KERNEL_PLAIN, True)
    assert (w * h == 1 or len(np.unique(want[0].reshape(-1, 4), axis=0)) > 8)
    for kernel in (abi.KERNEL_PLAIN, abi.KERNEL_AUTO):
        got = trace(kernel, False)
        assert np.array_equal(got[0], want[0])
        assert np.array_equal(fbits(got[1]), fbits(want[1]))
        assert got[2].tobytes() == want[2].tobytes()
