"""Steps launched behind one another without a wait on the host: a step's
kernel starts while the one before it still runs and waits for it on the
device.  The result equals that of the same steps with the host waiting after
each, and that of a captured graph of them, bit for bit (the kernel's sums do
not depend on the order of its blocks, so no tolerance is needed).
"""
import ctypes

import pytest

from entropicthreadsafe_b200 import capi, workloads
from test_zz_no_alloc import to_device_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (8, 24, 64, 100))
@pytest.mark.parametrize("mode", (capi.MODE_COLOUR, capi.MODE_PHASEFIELD, capi.MODE_SINGLE))
def test_back_to_back_steps_equal_separate_and_captured(n, mode):
    import torch
    p, f = workloads.droplet(n=n, radius=n / 4)
    p.mode = mode
    if mode == capi.MODE_PHASEFIELD:
        p.sharp_c = 0.9
        f["phi"] = 0.5 * (1 + f["phi"])
    if mode == capi.MODE_SINGLE:
        f["phi"][:] = 1.0
    stride = (n ** 3 + 31) // 32 * 32
    start = to_device_layout(f, stride)
    L = capi.lib()

    def steps(wait=False):
        bufs = [start.clone(), start.clone()]   # (the single-component step does not write phi)
        for k in range(12):
            rc = L.tslb_step_noalloc(ctypes.addressof(p), n, n, n, ctypes.c_void_p(bufs[k % 2].data_ptr()),
                                     ctypes.c_void_p(bufs[(k + 1) % 2].data_ptr()), stride,
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == capi.OK, L.tslb_last_error(None).decode()
            if wait:
                torch.cuda.synchronize()
        return bufs[0][:, :n ** 3]

    ref = steps(wait=True).clone()
    for _ in range(4):
        assert torch.equal(steps(), ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = steps()
    side.synchronize()
    assert torch.equal(got, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = steps()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
