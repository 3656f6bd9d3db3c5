"""The fused mixed kernel's tile plan with few screening spheres, which share
the threads (GPU): nuclei far apart, each with one s shell that reaches one
point only, so that a point left out of the tests loses that point's orbitals.
Sphere counts at the edges of 8, 4, 2 and 1 threads per sphere; the mixed form
against the FP64 form, within the mixed bound."""
import numpy as np
import pytest
import torch

from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 32, 33, 64, 65, 127, 128, 129, 250])
@pytest.mark.parametrize("comps", [1, 5])
def test_every_point_is_tested(n, comps):
    m = 16
    rng = np.random.default_rng(n)
    xyz = 8.0 * np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    one = np.ones(n, dtype=np.int64)
    d = dict(nucl_num=n, charge=np.ones(n), nucl_coord=np.ascontiguousarray(xyz.T), nucleus_index=np.arange(n),
             nucleus_shell_num=one, shell_ang_mom=np.zeros(n, dtype=np.int32), shell_prim_num=one,
             shell_prim_index=np.arange(n), shell_factor=np.ones(n), exponent=np.full(n, 5.0), coefficient=np.ones(n),
             prim_factor=np.ones(n), ao_factor=np.ones(n), ao_num=n, mo_num=m, mo_coef=rng.standard_normal((m, n)))
    pts = (xyz + 0.3 * rng.standard_normal((n, 3)))[rng.permutation(n)]
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    f = pq.b200_mo_vgl_device if comps == 5 else pq.b200_mo_value_device
    res = []
    for form in (pq.FORM_FP64, pq.FORM_MIXED):
        out = torch.full((n, comps, m), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx = make_context(d, points=False, form=form)
        try:
            f(ctx, n, c.data_ptr(), out.data_ptr())
            pq.b200_synchronize(ctx)
        finally:
            pq.context_destroy(ctx)
        res.append(out)
    ref, got = res
    assert bool((ref[:, 0].abs().amax(1) > 0).all())
    for k in range(comps):
        assert float((got[:, k] - ref[:, k]).abs().max()) <= 1e-6 * float(ref[:, k].abs().max())
