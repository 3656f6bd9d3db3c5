"""Calls queued one behind the other on a context's non-blocking stream, with
the nuclei or the MO coefficients changed between them and no synchronisation:
each call uses the inputs that were set when it was made (GPU).

A spinning kernel holds the stream back, so that every call is queued before
the first one starts.  The AO Hessian and the MO arrays are sums in a fixed
order and compared bit by bit with results of synchronised calls; the adjoint's
dL/dR is summed by atomics (1e-13 of the largest entry).
"""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu

P = 700


def _case(m):
    d = gen.config(0, walk_num=1)
    rng = np.random.default_rng(40 + m)
    d["mo_coef"] = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((d["ao_num"], m)))[0].T)
    d["mo_num"] = m
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1)
    pts = xyz.T[rng.integers(0, xyz.shape[1], P)] + rng.standard_normal((P, 3))
    geometries = [xyz, xyz + 0.3 * rng.standard_normal(xyz.shape), xyz - 0.2]
    coefs = [d["mo_coef"], np.ascontiguousarray(d["mo_coef"][::-1]), 2.0 * d["mo_coef"]]
    return d, pts, geometries, coefs, rng.standard_normal((P, 5, m))


def _outputs(d, call, m):
    e = lambda *s: torch.full(s, float("nan"), dtype=torch.float64, device="cuda")  # noqa: E731
    if call == "ao_hessian":
        return [e(3, P, 4, d["ao_num"])]
    if call == "adjoint":
        return [e(m, d["ao_num"]), e(d["nucl_num"], 3), e(3, P)]
    return [e(P, 5, m)]


def _queue(ctx, call, c, w, out):
    if call == "ao_hessian":
        pq.b200_ao_hessian_device(ctx, P, c.data_ptr(), out[0].data_ptr())
    elif call == "adjoint":
        pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), *(o.data_ptr() for o in out))
    else:
        pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), out[0].data_ptr())


@pytest.mark.parametrize("call,form,change,m", [
    ("ao_hessian", pq.FORM_FP64, "nuclei", 20), ("mo_vgl", pq.FORM_FP64, "nuclei", 20),
    ("mo_vgl", pq.FORM_FP64, "coefficients", 21), ("mo_vgl", pq.FORM_FP64, "coefficients", 20),
    ("adjoint", pq.FORM_FP64, "nuclei", 21), ("adjoint", pq.FORM_FP64, "coefficients", 21),
    ("adjoint", pq.FORM_MIXED, "nuclei", 21), ("adjoint", pq.FORM_MIXED, "coefficients", 21),
    ("mo_vgl", pq.FORM_MIXED, "nuclei", 20), ("mo_vgl", pq.FORM_MIXED, "coefficients", 21)])
def test_queued_calls_keep_their_inputs(call, form, change, m):
    d, pts, geometries, coefs, w = _case(m)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    c, dw = t(pts.T), t(w)
    ctx = make_context(d, points=False, form=form)
    stream = torch.cuda.Stream()
    pq.b200_set_stream(ctx, stream.cuda_stream)

    def set_input(i):
        if change == "nuclei":
            pq.set_nucleus_coord(ctx, "T", np.ascontiguousarray(geometries[i]).reshape(-1))
        else:
            pq.set_mo_basis_coefficient(ctx, np.ascontiguousarray(coefs[i]).reshape(-1))

    want, got = ([_outputs(d, call, m) for _ in range(3)] for _ in range(2))
    torch.cuda.synchronize()
    try:
        for i in range(3):
            set_input(i)
            _queue(ctx, call, c, dw, want[i])
            pq.b200_synchronize(ctx)
            torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(200_000_000)   # ~0.1 s
        for i in range(3):
            set_input(i)
            _queue(ctx, call, c, dw, got[i])
        busy = not stream.query()
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    if change == "nuclei" and (call, form) != ("mo_vgl", pq.FORM_MIXED):   # its tables are laid out anew
        assert busy   # a nuclear move does not wait for the stream
    for i in range(3):
        for a, b in zip(want[i], got[i]):
            if call == "adjoint":
                assert float((a - b).abs().max()) <= 1e-13 * float(a.abs().max())
            else:
                assert torch.equal(a, b)
    assert not torch.equal(want[0][-1], want[1][-1])
