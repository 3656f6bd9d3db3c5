"""AO Hessian (ao_hessian.cu) and bfloat16 AO pieces (ao_kernels.cu), GPU.

The AO Hessian goes by segments of at most 256 AOs, whose rows leave in bulk
copies from the 16-byte phase that they have in the output: odd and even AO
counts, one segment and several, an output that starts 8 bytes past a 16-byte
boundary, few points and more items than resident CTAs; against the oracle at
the FP64 bar, 1e-12.
The pieces feed dL/dC of the mixed adjoint alone.  Few points have their
nucleus blocks spread over warps: few and many points, AO counts that are no
multiple of 8; against the FP64 form, with the bound of the FP32 exponentials
and of the three-piece products (test_gpu_adjoint.py).
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


def _setup(cid, P, drop):
    d = gen.high_l_config(1) if cid == "hl" else gen.config(cid, walk_num=1)
    if drop:   # without the last nucleus
        s0, k0 = d["nucleus_index"][-1], d["shell_prim_index"][d["nucleus_index"][-1]]
        lmom = d["shell_ang_mom"][s0:]
        a = d["ao_num"] - int(((lmom + 1) * (lmom + 2) // 2).sum())
        for k in ("nucleus_index", "nucleus_shell_num", "charge"):
            d[k] = d[k][:-1]
        for k in ("shell_ang_mom", "shell_prim_num", "shell_prim_index", "shell_factor"):
            d[k] = d[k][:s0]
        for k in ("exponent", "coefficient", "prim_factor"):
            d[k] = d[k][:k0]
        d["nucl_num"] -= 1
        d["nucl_coord"] = np.ascontiguousarray(d["nucl_coord"][:, :-1])
        d["ao_factor"], d["ao_num"] = d["ao_factor"][:a], a
        d["mo_coef"] = np.ascontiguousarray(d["mo_coef"][:, :a])
    rng = np.random.default_rng(P)
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    return d, xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("cid,drop,P", [(0, 0, 1), (0, 1, 33), (0, 1, 2500), ("hl", 0, 7), (1, 1, 40), (4, 0, 3)])
def test_hessian(cid, drop, P, shift):
    d, pts = _setup(cid, P, drop)
    A = d["ao_num"]
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    buf = torch.full((12 * P * A + 2,), float("nan"), dtype=torch.float64, device="cuda")
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        torch.cuda.synchronize()
        pq.b200_ao_hessian_device(ctx, P, c.data_ptr(), buf.data_ptr() + 8 * shift)
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    got = buf.cpu().numpy()
    assert np.isnan(got[:shift]).all() and np.isnan(got[12 * P * A + shift:]).all()
    got = got[shift:12 * P * A + shift].reshape(3, P, 4, A)
    assert parity_error(got, O.ao_hessian(O.Basis(d), pts, d["nucl_coord"])) < 1e-12


@pytest.mark.parametrize("cid,drop,P", [(0, 0, 1), (0, 1, 31), (0, 0, 32), (0, 1, 33), ("hl", 0, 40), (1, 1, 70),
                                        (0, 1, 5000)])
def test_pieces(cid, drop, P):
    d, pts = _setup(cid, P, drop)
    m = d["mo_coef"].shape[0]
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, w = t(pts.T), t(np.random.default_rng(P + 1).standard_normal((P, 5, m)))
    res = []
    for form in (pq.FORM_FP64, pq.FORM_MIXED):
        ctx = make_context(d, points=False, form=form)
        g = torch.full((m, d["ao_num"]), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        try:
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), g.data_ptr(), 0, 0)
            pq.b200_synchronize(ctx)
        finally:
            pq.context_destroy(ctx)
        res.append(g)
    assert float((res[1] - res[0]).abs().max()) <= 1e-6 * float(res[0].abs().max())
