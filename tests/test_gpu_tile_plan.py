"""The fused mixed kernel's tile plan where its spheres take several passes,
with spread and with coincident points and a NaN point (GPU): the mixed form
against the FP64 form, within the mixed bound per component."""
import numpy as np
import pytest
import torch

from conftest import comp_error
from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu

MIXED_TOL = 1e-6


@pytest.mark.parametrize("points", ["spread", "one", "same", "nan"])
def test_many_shells(points):
    rng = np.random.default_rng(31)
    charges = [6.0] * 150 + [1.0] * 150
    xyz = gen.place_nuclei(rng, 300, 40.0)
    d = gen.build_system(rng, charges, xyz, gen.SHAPES["tz_heavy"], gen.SHAPES["tz_h"], 20, 1, elec_num=2)
    assert d["shell_ang_mom"].size > 2048
    pts = xyz[rng.integers(0, 300, 90)] + rng.standard_normal((90, 3))
    if points == "one":
        pts = pts[:1]
    if points == "same":
        pts[:] = pts[0]
    keep = np.ones(pts.shape[0], dtype=bool)
    if points == "nan":
        pts[40, 2] = np.nan
        keep[40] = False
    P = pts.shape[0]
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    out = {}
    for form in (pq.FORM_FP64, pq.FORM_MIXED):
        ctx = make_context(d, points=False, form=form)
        o = torch.empty((P, 5, 20), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), o.data_ptr())
        pq.b200_synchronize(ctx)
        pq.context_destroy(ctx)
        out[form] = o.cpu().numpy()[keep]
    assert max(comp_error(out[pq.FORM_MIXED], out[pq.FORM_FP64])) < MIXED_TOL
