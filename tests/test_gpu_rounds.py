"""The wavefront's automatic choice between rounds and the finishing kernel
alone: no round on triangle-only scenes whose rays are short (by the BVH's
estimate) at any frame size, rounds on the others; the same bits either way,
for a frame, a batch and an adjoint."""
import numpy as np
import pytest

from conftest import fbits

from gpu_cases import soup_scene
from vktrace import abi
from vktrace import scene as S

pytestmark = pytest.mark.gpu

NEVER = 1  # tail_paths: rounds to the end


def _params(w, h, tail, **kw):
    return abi.Tracer.params(w, h, spp=2, max_depth=4, rr_start=2, sky=(1.0, 0.9, 0.8), kernel=abi.KERNEL_WAVEFRONT,
                             tail_paths=tail, aovs=(abi.AOV_RGBA32F, abi.AOV_LINEAR), **kw)


@pytest.mark.parametrize("n,extent,planes,rounds", [
    (1, 10.0, False, False),        # a single triangle
    (1500, 10.0, False, False),
    (1500, 10.0, True, False),      # with a plane: tested after the triangles
    (40_000, 50.0, False, True),    # long rays
])
def test_rounds_only_for_long_rays(gpu_tracer, n, extent, planes, rounds):
    tr = gpu_tracer
    sc = soup_scene(71, n, extent=extent, sigma=0.01 * extent)
    if planes:
        sc.planes = np.zeros(1, S.PLANE)
        sc.planes[0]["mat"] = S.material((0.8, 0.7, 0.6), roughness=0.4)
        sc.planes[0]["N"], sc.planes[0]["len"] = (0.0, 1.0, 0.0), 12.0
    tr.upload_scene(sc)
    w, h = 641, 463  # more paths than twice the resident threads
    fr = S.frame(S.look_at((0.0, 0.1 * extent, 2.4 * extent), (0.0, 0.0, 0.0), 40.0), w / h, 0.4)
    tr.trace(fr, _params(w, h, 0))
    got = tr.readback(abi.AOV_RGBA32F)
    assert (tr_rounds(tr, fr, w, h) > 0) == rounds
    tr.trace(fr, _params(w, h, NEVER))
    assert np.array_equal(fbits(got), fbits(tr.readback(abi.AOV_RGBA32F)))
    lin = tr.readback(abi.AOV_LINEAR)
    dl = np.random.default_rng(2).standard_normal((h, w, 4)).astype(np.float32)
    grads = [tr.trace_adjoint(fr, _params(w, h, tail), dl, lin, num_materials=len(sc.materials))
             for tail in (0, NEVER)]
    for a, b in zip(*grads):  # FP64 sums in another order
        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-7 * max(1e-30, float(np.max(np.abs(b)))))


def tr_rounds(tr, fr, w, h):
    tr.set_profiling(True)
    try:
        tr.trace(fr, _params(w, h, 0))
        return tr.timings()["rounds"]
    finally:
        tr.set_profiling(False)


def test_batch_of_short_rays(gpu_tracer):
    """A batch takes the pixel-weighted mean of its scenes' estimates."""
    tr = gpu_tracer
    scenes = [soup_scene(80, 900), soup_scene(81, 1), soup_scene(82, 3000, extent=20.0, sigma=0.2)]
    sizes = [(400, 300), (31, 17), (500, 331)]
    frames = [S.frame(S.look_at((1.0 * i, 2.0, 40.0), (0.0, 0.0, 0.0), 40.0), w / h, 0.1 * i)
              for i, (w, h) in enumerate(sizes)]
    tr.upload_scenes(scenes)
    imgs = []
    for tail, graph in ((0, False), (0, True), (NEVER, False)):
        params = [_params(w, h, tail) for w, h in sizes]
        for p in params:
            p.aov_mask = 1 << abi.AOV_RGBA32F
        tr.trace_batched(frames, params, use_graph=graph)
        imgs.append([tr.readback_scene(i, abi.AOV_RGBA32F).copy() for i in range(len(scenes))])
    for other in imgs[1:]:
        for a, b in zip(imgs[0], other):
            assert np.array_equal(fbits(a), fbits(b))
