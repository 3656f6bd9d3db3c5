"""Loss weights that are not finite (GPU): the adjoint is linear in the
weights, and an infinite or NaN weight times an AO that is exactly zero is a
NaN, so the gradients that hold the product are not finite: dL/dC of the MO,
dL/dR of every nucleus and dL/dr of the point.  Everything else is the
gradient without that weight.  The point lies beyond the reach of all AOs (an
electron far out, whose orbitals vanish and whose 1 / psi overflows), or at one
side of a molecule whose other side does not reach it, among points that are
reached.
"""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


def _grads(ctx, d, pts, w):
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw, P = t(pts.T), t(w), pts.shape[0]
    out = [torch.empty(s, dtype=torch.float64, device="cuda")
           for s in ((d["mo_num"], d["ao_num"]), (d["nucl_num"], 3), (3, P))]
    torch.cuda.synchronize()
    pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), dw.data_ptr(), *(o.data_ptr() for o in out))
    pq.b200_synchronize(ctx)
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("form,tol", [(pq.FORM_FP64, 1e-13), (pq.FORM_MIXED, 1e-6)])
@pytest.mark.parametrize("value,comp,mo", [(np.inf, 0, 0), (-np.inf, 4, 89), (np.nan, 2, 37)])
@pytest.mark.parametrize("cid,P", [(0, 20), (0, 700), (0, 40000), (1, 300)])
def test_a_weight_that_is_not_finite(form, tol, value, comp, mo, cid, P):
    d = gen.config(cid, walk_num=1)
    rng = np.random.default_rng(3)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    pts = xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))
    bad = P // 3
    pts[bad] = xyz.max(0) + 60.0 if cid == 0 else xyz[np.argmax(xyz[:, 0])]
    w = rng.standard_normal((P, 5, d["mo_num"]))
    w[bad] = 0.0
    ctx = make_context(d, points=False, form=form)
    try:
        clean = _grads(ctx, d, pts, w)
        w[bad, comp, mo] = value
        gc, gn, gr = _grads(ctx, d, pts, w)
    finally:
        pq.context_destroy(ctx)
    assert not np.isfinite(gc[mo]).any()
    assert not np.isfinite(gn).any()
    assert not np.isfinite(gr[:, bad]).any()
    others = np.arange(d["mo_num"]) != mo
    rest = np.arange(P) != bad
    for a, b in ((gc[others], clean[0][others]), (gr[:, rest], clean[2][:, rest])):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
