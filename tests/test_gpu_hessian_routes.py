"""The two forms of the AO Hessian kernel, images of AO segments and a warp per
point, at the point counts where the dispatch changes between them (GPU): many
points in one call, which take a warp each, give the bits of calls of a few
hundred, which take images.  Odd row lengths and output addresses, FP32
exponentials (precision of 23 bits), and the cusp adjustment's masked AOs
through the MO Hessian; a part of the points against the oracle."""
import numpy as np
import pytest
import torch

from conftest import parity_error
from oracle import pyoracle as O
from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context
from test_oracle_cusp import cusp_system, near_nuclei

pytestmark = pytest.mark.gpu


def _molecule(kind):
    if kind == "hl":
        return gen.high_l_config(1)
    if kind == "config0":
        return gen.config(0, walk_num=1)
    rng = np.random.default_rng(17)
    n = int(kind)
    return gen.build_system(rng, [6.0] * (n - 1) + [1.0], gen.place_nuclei(rng, n, 8.0), gen.SHAPES["tz_heavy"],
                            gen.SHAPES["tz_h"], 4, 1, elec_num=2)


def _hessian(ctx, pts, A, shift):
    P = pts.shape[0]
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    buf = torch.full((12 * P * A + 2,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    pq.b200_ao_hessian_device(ctx, P, c.data_ptr(), buf.data_ptr() + 8 * shift)
    pq.b200_synchronize(ctx)
    assert bool(torch.isnan(buf[:shift]).all()) and bool(torch.isnan(buf[12 * P * A + shift:]).all())
    return buf[shift:12 * P * A + shift].reshape(3, P, 4, A)


@pytest.mark.parametrize("kind,P,piece", [("config0", 1000, 250), ("config0", 1003, 400), ("1", 1001, 333),
                                          ("6", 2100, 700), ("hl", 5001, 1667), ("10", 700, 350)])
@pytest.mark.parametrize("precision", [53, 23])
@pytest.mark.parametrize("shift", [0, 1])
def test_routes_agree(kind, P, piece, precision, shift):
    d = _molecule(kind)
    A = d["ao_num"]
    rng = np.random.default_rng(P)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    pts = xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))
    pts[5] = [np.nan, 0.0, 0.0]
    pts[6] = [np.inf, 0.0, 0.0]
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        pq.set_numprec_precision(ctx, precision)
        got = _hessian(ctx, pts, A, shift)
        parts = torch.cat([_hessian(ctx, pts[a:a + piece], A, shift) for a in range(0, P, piece)], 1)
    finally:
        pq.context_destroy(ctx)
    assert torch.equal(got.nan_to_num(nan=-1.5), parts.nan_to_num(nan=-1.5))
    assert bool(torch.isnan(got[:, 5]).any()) and bool((got[:, 6] == 0.0).all())
    if precision == 53:
        ref = O.ao_hessian(O.Basis(d), pts[10:60], d["nucl_coord"])
        assert parity_error(got[:, 10:60].cpu().numpy(), ref) < 1e-12


def test_routes_agree_with_cusp():
    d, rc = cusp_system()
    M = d["mo_num"]
    pts = np.concatenate([near_nuclei(d, rc, per=6, seed=s) for s in range(30)])[:1200]
    assert pts.shape[0] >= 1000
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    res = []
    try:
        pq.set_mo_basis_r_cusp(ctx, rc)
        for part in [pts] + [pts[a:a + 400] for a in range(0, pts.shape[0], 400)]:
            n = part.shape[0]
            pq.set_point(ctx, "N", n, np.ascontiguousarray(part).reshape(-1))
            res.append(pq.get_mo_basis_mo_hessian(ctx, 9 * n * M).reshape(3, n, 3, M))
    finally:
        pq.context_destroy(ctx)
    # the contraction's row blocks differ with the count: the bar of the FP64 form
    assert parity_error(res[0], np.concatenate(res[1:], 1)) < 1e-12
