"""The mixed adjoint with all AOs per tile (up to 2 million point-AO pairs) and
with the tiles' lists above (GPU): a count just above that line against calls of a few hundred of its
points, and all AOs against the FP64 form within the mixed adjoint's bound, also
with a point whose weights are not finite.  The derivative kernel's tiles are
shared by up to 24 CTAs where there are many shells."""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


def _grads(d, pts, w, form):
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw, P = t(pts.T), t(w), pts.shape[0]
    gn, gr = (torch.full(s, float("nan"), dtype=torch.float64, device="cuda") for s in ((d["nucl_num"], 3), (3, P)))
    torch.cuda.synchronize()
    ctx = make_context(d, points=False, form=form)
    try:
        pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), dw.data_ptr(), 0, gn.data_ptr(), gr.data_ptr())
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    return gn, gr


def _case(cid, P):
    d = gen.high_l_config(1) if cid == "hl" else gen.config(cid, walk_num=1)
    rng = np.random.default_rng(P)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    return d, xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3)), rng.standard_normal((P, 5, d["mo_num"]))


# the first counts with lists: 22,223 points of 90 AOs, 4,567 of 438, 1,001 of 2000
@pytest.mark.parametrize("cid,P", [(0, 22223), ("hl", 4567), (1, 1001)])
def test_both_sides_of_the_line(cid, P):
    d, pts, w = _case(cid, P)
    assert 2_000_000 < P * d["ao_num"] <= 2_000_000 + d["ao_num"]
    lists = _grads(d, pts, w, pq.FORM_MIXED)
    parts = [_grads(d, pts[a:a + 777], w[a:a + 777], pq.FORM_MIXED) for a in range(0, P, 777)]   # with all AOs
    gn, gr = sum(p[0] for p in parts), torch.cat([p[1] for p in parts], 1)
    # the same products, summed in FP64 in another order
    for a, b in zip(lists, (gn, gr)):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())


@pytest.mark.parametrize("cid,P", [(0, 1), (0, 32), (0, 33), (0, 1000), (1, 70)])
def test_all_aos_against_fp64(cid, P):
    d, pts, w = _case(cid, P)
    got, ref = _grads(d, pts, w, pq.FORM_MIXED), _grads(d, pts, w, pq.FORM_FP64)
    for a, b in zip(got, ref):
        assert float((a - b).abs().max()) <= 1e-6 * float(b.abs().max())
    w[P // 2, 1, 0] = np.inf
    gn, gr = _grads(d, pts, w, pq.FORM_MIXED)
    assert not bool(torch.isfinite(gr[:, P // 2]).any()) and not bool(torch.isfinite(gn).any())
    rest = torch.arange(P, device="cuda") != P // 2
    assert torch.equal(gr[:, rest], got[1][:, rest])
