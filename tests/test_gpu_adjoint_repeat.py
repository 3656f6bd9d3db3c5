"""dL/dr is summed in a fixed order, also where several blocks share a tile of
points: the same bits in every run (GPU)."""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [pq.FORM_FP64, pq.FORM_MIXED])
@pytest.mark.parametrize("cid,P", [(0, 20), (0, 700), (1, 1000), (0, 14000), (0, 15000), (0, 30000)])
def test_point_gradient_repeats(form, cid, P):
    d = gen.config(cid, walk_num=1)
    rng = np.random.default_rng(P)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    pts = xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, w = t(pts.T), t(rng.standard_normal((P, 5, d["mo_num"])))
    out = [torch.full((3, P), float("nan"), dtype=torch.float64, device="cuda") for _ in range(6)]
    torch.cuda.synchronize()
    ctx = make_context(d, points=False, form=form)
    try:
        for o in out:
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), 0, 0, o.data_ptr())
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    assert bool(torch.isfinite(out[0]).all()) and float(out[0].abs().max()) > 0.0
    assert all(torch.equal(out[0], o) for o in out[1:])
