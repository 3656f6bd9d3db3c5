"""An FP64 evaluation that needs more scratch while its stream is captured fails
(device memory cannot be allocated there), and the context then evaluates as
before: the failed allocation is not taken for a full device, which would leave
it with small chunks (GPU)."""
import ctypes

import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


def test_a_capture_does_not_shrink_the_chunks():
    d = gen.config(0, walk_num=1)
    P, M = 9000, d["mo_num"]
    rng = np.random.default_rng(2)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    pts = xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))
    c = torch.tensor(np.ascontiguousarray(pts.T), device="cuda")
    values = torch.empty((P, M), dtype=torch.float64, device="cuda")
    out = torch.empty((P, 5, M), dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def launches(ctx):
        n0 = pq.b200_kernel_launch_count()
        pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), out.data_ptr())
        pq.b200_synchronize(ctx)
        return pq.b200_kernel_launch_count() - n0

    fresh = make_context(d, points=False, form=pq.FORM_FP64)
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        want = launches(fresh)
        ref = out.clone()
        pq.b200_set_stream(ctx, stream.cuda_stream)
        pq.b200_mo_value_device(ctx, P, c.data_ptr(), values.data_ptr())   # tables, order, a fifth of the scratch
        pq.b200_synchronize(ctx)
        # by the runtime itself: torch's allocator would take the capture that fails for one that goes on
        rt = ctypes.CDLL("libcudart.so.12")
        s, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
        assert rt.cudaStreamBeginCapture(s, 1) == 0   # thread-local
        try:
            with pytest.raises(RuntimeError):
                pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), out.data_ptr())
        finally:
            rt.cudaStreamEndCapture(s, ctypes.byref(graph))   # the capture was invalidated
            if graph.value:
                rt.cudaGraphDestroy(graph)
            rt.cudaGetLastError()
        torch.cuda.synchronize()
        out.fill_(float("nan"))
        assert launches(ctx) == want
        assert torch.equal(out, ref)
    finally:
        pq.context_destroy(ctx)
        pq.context_destroy(fresh)
