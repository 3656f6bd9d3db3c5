"""The FP64 evaluations on a device with little memory left (GPU): their
scratch of up to 4 GiB gives way to smaller chunks of points instead of a
failed allocation.  The forward's results are the same bits, the gradients'
sums run over other chunks (1e-13 of the largest entry)."""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


def test_scratch_gives_way():
    P = 20352
    d = gen.config(1, walk_num=1)
    rng = np.random.default_rng(8)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    pts = xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))
    e = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")  # noqa: E731
    c = torch.tensor(np.ascontiguousarray(pts.T), device="cuda")
    w = torch.tensor(rng.standard_normal((P, 5, d["mo_num"])), device="cuda")
    outs = [[e(P, 5, d["mo_num"]), e(d["mo_num"], d["ao_num"]), e(d["nucl_num"], 3), e(3, P)] for _ in range(3)]
    torch.cuda.synchronize()
    hold = None
    for i in range(3):
        if i == 1:   # 0.7 GiB left; in turn 2 the calls come again
            torch.cuda.empty_cache()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - 700 * 2**20, dtype=torch.uint8, device="cuda")
        if i < 2:
            ctx = make_context(d, points=False, form=pq.FORM_FP64)
        o = outs[i]
        try:
            pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), o[0].data_ptr())
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), *(x.data_ptr() for x in o[1:]))
            pq.b200_synchronize(ctx)
        finally:
            if i != 1:
                pq.context_destroy(ctx)
    del hold
    torch.cuda.empty_cache()
    for o in outs[1:]:
        assert torch.equal(o[0], outs[0][0])
        for a, b in zip(o[1:], outs[0][1:]):
            assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())
