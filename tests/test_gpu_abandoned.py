"""A call that gives up waiting for its own queue lengths (a short time limit)
leaves kernels running that will still report a ray over the step limit.  The
next call waits for them and returns its own status and image."""
import numpy as np
import pytest
import torch

from vktrace import abi, configs

pytestmark = pytest.mark.gpu

SIDE = 4096  # 16.8 M paths: the first round takes longer than the time limit


@pytest.mark.parametrize("call", ["trace", "batch", "adjoint"])
def test_status_of_an_abandoned_call_is_not_the_next_ones(tracer_lib, call):
    wl = configs.c1()
    big = abi.Tracer.params(SIDE, SIDE, spp=2, max_depth=8, rr_start=wl.rr_start, sky=wl.sky, tail_paths=1,
                            kernel=abi.KERNEL_WAVEFRONT, aovs=(abi.AOV_RGBA8,))
    small = abi.Tracer.params(160, 90, spp=2, max_depth=4, rr_start=wl.rr_start, sky=wl.sky)
    with abi.Tracer(0) as tr:
        tr.upload_scene(wl.scene)
        if call == "batch":
            tr.upload_scenes([wl.scene])
        zeros = torch.zeros((SIDE, SIDE, 4), device="cuda")
        torch.cuda.synchronize()
        tr.trace(wl.frame, small)
        want = tr.readback(abi.AOV_RGBA8)
        tr.set_traversal_limit(60)  # the mean ray visits 36 nodes
        tr.set_timeout(1)
        with pytest.raises(abi.TracerError) as e:
            if call == "trace":
                tr.trace(wl.frame, big)
            elif call == "batch":
                tr.trace_batched([wl.frame], [big], use_graph=False)
            else:
                tr.trace_adjoint(wl.frame, big, zeros.data_ptr(), zeros.data_ptr(),
                                 num_materials=len(wl.scene.materials))
        assert e.value.status == abi.ERR_TIMEOUT
        tr.set_timeout(60000)
        tr.set_traversal_limit(0)
        tr.trace(wl.frame, small)
        tr.synchronize()
        assert np.array_equal(tr.readback(abi.AOV_RGBA8), want)
