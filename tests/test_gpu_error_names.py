"""A failure in the tables that several calls share names the call that needed
them (GPU; the failing allocation is injected on the host)."""
import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call,name", [("ao_hessian", "qmckl_b200_ao_hessian"), ("mo_vgl", "qmckl_b200_mo_fp64"),
                                       ("adjoint", "qmckl_b200_mo_vgl_adjoint_device")])
def test_shell_records_name_their_caller(call, name):
    d = gen.config(0, walk_num=1)
    P, A, M = 4, d["ao_num"], d["mo_num"]
    e = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
    c, w, out = e(3, P), e(P, 5, M), [e(max(12 * P * A, M * A)), e(d["nucl_num"], 3), e(3, P)]
    torch.cuda.synchronize()
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        pq.b200_ao_vgl_device(ctx, P, c.data_ptr(), out[0].data_ptr())   # the basis is on the device
        pq.b200_synchronize(ctx)
        pq.b200_inject_alloc_failure(0)
        with pytest.raises(RuntimeError, match=name):
            if call == "ao_hessian":
                pq.b200_ao_hessian_device(ctx, P, c.data_ptr(), out[0].data_ptr())
            elif call == "adjoint":
                pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), *(o.data_ptr() for o in out))
            else:
                pq.b200_mo_vgl_device(ctx, P, c.data_ptr(), out[0].data_ptr())
    finally:
        pq.b200_inject_alloc_failure(-1)
        pq.context_destroy(ctx)
    assert np.isfinite(out[0].cpu().numpy()).all()
