"""FP64 MO evaluation over compact spatial tiles (f64_tiles.cu) at the edges
of its tiles and of its dispatch, against the oracle (GPU).

VGL tiles hold 32 points and value tiles 32 or, from 75,776 points on, 128;
the contraction takes 80-column tiles once there are four CTAs per SM of them
and narrower ones below; a tile's AO list is staged 1024 entries at a time;
more than 1024 shells are numbered by another pass; up to 4096 points are put
in order by one CTA.  The bar is the parity
bar of the FP64 form (1e-12, tests/conftest.py).
"""
import numpy as np
import pytest
import torch

from conftest import parity_error
from oracle import pyoracle as O
from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _molecule(cid, m, seed):
    d = gen.high_l_config(1) if cid == "hl" else gen.config(cid, walk_num=1)
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((d["ao_num"], m)))
    d["mo_coef"] = np.ascontiguousarray(q.T)
    d["mo_num"] = m
    return d


def _points(d, P, seed):
    rng = np.random.default_rng(seed)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    return xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))


def _device(ctx, pts, m, comps):
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    out = torch.full((pts.shape[0], comps, m), float("nan"), dtype=torch.float64, device="cuda")
    f = pq.b200_mo_vgl_device if comps == 5 else pq.b200_mo_value_device
    torch.cuda.synchronize()
    f(ctx, pts.shape[0], c.data_ptr(), out.data_ptr())
    pq.b200_synchronize(ctx)
    return out.cpu().numpy()


@pytest.mark.parametrize("cid,P,m,comps", [
    (0, 1, 1, 5), (0, 31, 33, 5), (0, 32, 64, 5), (0, 33, 81, 5), (0, 1300, 90, 5), (0, 4096, 20, 5), (0, 4097, 20, 5), (0, 9473, 90, 5),
    (0, 1, 1, 1), (0, 33, 31, 1), (0, 4736, 65, 1), (0, 75775, 17, 1), (0, 75777, 81, 1),
    ("hl", 70, 120, 5), ("hl", 70, 101, 1), (1, 32, 160, 5), (4, 32, 350, 5), (4, 40, 33, 1)])
def test_tiles(cid, P, m, comps):
    d = _molecule(cid, m, 100 + P)
    pts = _points(d, P, 200 + P)
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        got = _device(ctx, pts, m, comps)
    finally:
        pq.context_destroy(ctx)
    if comps == 5:
        ref = O.mo_vgl(d["mo_coef"], O.ao_vgl(O.Basis(d), pts, d["nucl_coord"]))
    else:
        ref = O.mo_value(d["mo_coef"], O.ao_value(O.Basis(d), pts, d["nucl_coord"])).reshape(P, 1, m)
    assert parity_error(got, ref) < TOL


def test_nan_point_stays_alone():
    d = _molecule(0, 90, 5)
    pts = _points(d, 100, 6)
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        bad = pts.copy()
        bad[17, 1] = np.nan
        got = _device(ctx, bad, 90, 5)
        far = pts.copy()
        far[17] = [np.inf, 0.0, 0.0]
        got_far = _device(ctx, far, 90, 5)
    finally:
        pq.context_destroy(ctx)
    ref = O.mo_vgl(d["mo_coef"], O.ao_vgl(O.Basis(d), pts, d["nucl_coord"]))
    keep = np.arange(100) != 17
    assert np.isnan(got[17]).any()
    assert parity_error(got[keep], ref[keep]) < TOL
    assert (got_far[17] == 0.0).all()
    assert parity_error(got_far[keep], ref[keep]) < TOL


@pytest.mark.parametrize("cid,P,m", [(0, 1, 3), (0, 32, 90), (0, 33, 81), (0, 100, 17), ("hl", 40, 101), (1, 50, 33)])
def test_adjoint_tiles(cid, P, m):
    """dL/dC, dL/dR and dL/dr over the tiles, against the oracle (the bar of test_gpu_adjoint.py)."""
    d = _molecule(cid, m, 300 + P)
    pts = _points(d, P, 400 + P)
    w = np.random.default_rng(500 + P).standard_normal((P, 5, m))
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw = t(pts.T), t(w)
    nan = float("nan")
    gc, gn, gr = (torch.full(s, nan, dtype=torch.float64, device="cuda")
                  for s in ((m, d["ao_num"]), (d["nucl_num"], 3), (3, P)))
    torch.cuda.synchronize()
    try:
        pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), dw.data_ptr(), gc.data_ptr(), gn.data_ptr(), gr.data_ptr())
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    ref = O.mo_vgl_adjoint(O.Basis(d), pts, d["nucl_coord"], d["mo_coef"], w)
    for got, want in zip((gc, gn, gr.T), ref):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-10 * np.abs(want).max()


@pytest.mark.parametrize("cid,P,m", [(0, 1, 3), (0, 32, 64), (0, 33, 81), (0, 100, 17), ("hl", 40, 101), (1, 50, 161),
                                     (0, 12000, 20)])
def test_mixed_adjoint_tiles(cid, P, m):
    """The mixed adjoint's pulled-back weights over the tiles' AO lists, at the edges of their row blocks (128), K
    blocks (64 MOs) and tiles: against the FP64 form, within the mixed adjoint's bound (test_gpu_adjoint.py)."""
    d = _molecule(cid, m, 600 + P)
    pts = _points(d, P, 700 + P)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw = t(pts.T), t(np.random.default_rng(800 + P).standard_normal((P, 5, m)))
    res = []
    for form in (pq.FORM_FP64, pq.FORM_MIXED):
        ctx = make_context(d, points=False, form=form)
        gn, gr = (torch.full(s, float("nan"), dtype=torch.float64, device="cuda") for s in ((d["nucl_num"], 3), (3, P)))
        torch.cuda.synchronize()
        try:
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), dw.data_ptr(), 0, gn.data_ptr(), gr.data_ptr())
            pq.b200_synchronize(ctx)
        finally:
            pq.context_destroy(ctx)
        res.append((gn, gr))
    for ref, got in zip(*res):
        assert float((got - ref).abs().max()) <= 1e-6 * float(ref.abs().max())


def test_adjoint_coefficients_repeat():
    """dL/dC is summed in a fixed order: the same bits in every run."""
    d = _molecule(0, 90, 8)
    pts = _points(d, 5000, 9)
    w = torch.randn((5000, 5, 90), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    out = []
    torch.cuda.synchronize()
    try:
        for _ in range(3):
            g = torch.empty((90, d["ao_num"]), dtype=torch.float64, device="cuda")
            pq.b200_mo_vgl_adjoint_device(ctx, 5000, c.data_ptr(), w.data_ptr(), g.data_ptr(), 0, 0)
            pq.b200_synchronize(ctx)
            out.append(g)
    finally:
        pq.context_destroy(ctx)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


def test_adjoint_many_shells():
    """More shells than a tile's lists hold at a time (25,600): listed in windows."""
    n, per, P, m = 2600, 10, 40, 3
    rng = np.random.default_rng(11)
    S = n * per
    grid = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2.0
    d = dict(nucl_num=n, charge=np.ones(n), nucl_coord=np.ascontiguousarray(grid.T.astype(float)),
             nucleus_index=np.arange(0, S, per), nucleus_shell_num=np.full(n, per), shell_ang_mom=np.zeros(S, dtype=np.int32),
             shell_prim_num=np.ones(S, dtype=np.int64), shell_prim_index=np.arange(S), shell_factor=np.ones(S),
             exponent=rng.uniform(0.3, 20.0, S), coefficient=np.ones(S), prim_factor=np.ones(S), ao_factor=np.ones(S),
             ao_num=S, mo_num=m, mo_coef=rng.standard_normal((m, S)))
    # points around the nuclei on both sides of the window's edge (nucleus 2560)
    pts = grid[rng.integers(2400, n, P)] + rng.standard_normal((P, 3))
    w = rng.standard_normal((P, 5, m))
    ref = O.mo_vgl_adjoint(O.Basis(d), pts, d["nucl_coord"], d["mo_coef"], w)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw = t(pts.T), t(w)
    for form, tol in ((pq.FORM_FP64, 1e-10), (pq.FORM_MIXED, 1e-6)):
        ctx = make_context(d, points=False, form=form)
        gc, gn, gr = (torch.full(s, float("nan"), dtype=torch.float64, device="cuda") for s in ((m, S), (n, 3), (3, P)))
        torch.cuda.synchronize()
        try:
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), dw.data_ptr(), gc.data_ptr(), gn.data_ptr(), gr.data_ptr())
            pq.b200_synchronize(ctx)
        finally:
            pq.context_destroy(ctx)
        for got, want in zip((gc, gn, gr.T), ref):
            assert np.abs(got.cpu().numpy() - want).max() <= tol * np.abs(want).max()
