"""The tile plans of the fused mixed kernel and of the batched one with few
screening spheres, which share the threads (GPU): nuclei far apart, each with
one s shell that reaches one point only, so that a point left out of the tests
loses that point's orbitals.  Sphere counts at the edges of 8, 4, 2 and 1
threads per sphere; the mixed form against the FP64 form, within the mixed
bound."""
import numpy as np
import pytest
import torch

from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


M = 16


def _scattered(n):
    """n nuclei far apart with a tight s shell each, and a point near every nucleus, in another order."""
    rng = np.random.default_rng(n)
    xyz = 8.0 * np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    one = np.ones(n, dtype=np.int64)
    d = dict(nucl_num=n, charge=np.ones(n), nucl_coord=np.ascontiguousarray(xyz.T), nucleus_index=np.arange(n),
             nucleus_shell_num=one, shell_ang_mom=np.zeros(n, dtype=np.int32), shell_prim_num=one,
             shell_prim_index=np.arange(n), shell_factor=np.ones(n), exponent=np.full(n, 5.0), coefficient=np.ones(n),
             prim_factor=np.ones(n), ao_factor=np.ones(n), ao_num=n, mo_num=M, mo_coef=rng.standard_normal((M, n)))
    return d, (xyz + 0.3 * rng.standard_normal((n, 3)))[rng.permutation(n)]


def _single(d, pts, form, comps):
    n = pts.shape[0]
    c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
    out = torch.full((n, comps, M), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx = make_context(d, points=False, form=form)
    try:
        f = pq.b200_mo_vgl_device if comps == 5 else pq.b200_mo_value_device
        f(ctx, n, c.data_ptr(), out.data_ptr())
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    return out


def _agree(got, ref):
    assert bool((ref[:, 0].abs().amax(1) > 0).all())
    for k in range(ref.shape[1]):
        assert float((got[:, k] - ref[:, k]).abs().max()) <= 1e-6 * float(ref[:, k].abs().max())


@pytest.mark.parametrize("n", [8, 32, 33, 64, 65, 127, 128, 129, 250])
@pytest.mark.parametrize("comps", [1, 5])
def test_every_point_is_tested(n, comps):
    d, pts = _scattered(n)
    _agree(_single(d, pts, pq.FORM_MIXED, comps), _single(d, pts, pq.FORM_FP64, comps))


@pytest.mark.parametrize("producers", [8, 16])
def test_every_point_is_tested_in_a_batch(producers):
    systems = [_scattered(n) for n in (8, 33, 80, 81, 160, 161, 320, 321, 400)]
    ctxs = [make_context(d, points=False, form=pq.FORM_MIXED) for d, _ in systems]
    P = [x.shape[0] for _, x in systems]
    batch = pq.b200_batch_create(ctxs, P)
    try:
        pq.b200_batch_set_tuning(batch, producers, 0)
        co, oo, (ct, ot) = pq.b200_batch_layout(batch, len(P))
        coord = np.zeros(ct)
        for s, (_, x) in enumerate(systems):
            coord[co[s]:co[s] + 3 * P[s]] = np.ascontiguousarray(x.T).reshape(-1)
        c = torch.tensor(coord, device="cuda")
        out = torch.full((ot,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        pq.b200_batch_mo_vgl_device(batch, c.data_ptr(), out.data_ptr())
        pq.b200_batch_synchronize(batch)
    finally:
        pq.b200_batch_destroy(batch)
        for ctx in ctxs:
            pq.context_destroy(ctx)
    for s, (d, x) in enumerate(systems):
        got = out[oo[s]:oo[s] + P[s] * 5 * M].reshape(P[s], 5, M)
        _agree(got, _single(d, x, pq.FORM_FP64, 5))
