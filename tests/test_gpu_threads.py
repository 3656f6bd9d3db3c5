"""Contexts of different sizes used by several host threads at once, each on
its own stream (GPU): a kernel's shared-memory opt-in belongs to the process,
so that one thread's small molecule must not narrow it under another thread's
large one.  Every call succeeds and gives the bits of a call made alone.
"""
import threading

import numpy as np
import pytest
import torch

from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu

P, CALLS = 33, 4000


def _chain(n, per, m):
    """n nuclei in a row, `per` s shells each."""
    rng = np.random.default_rng(n)
    S = n * per
    xyz = np.zeros((3, n))
    xyz[0] = 1.5 * np.arange(n)
    return dict(nucl_num=n, charge=np.ones(n), nucl_coord=xyz, nucleus_index=np.arange(0, S, per),
                nucleus_shell_num=np.full(n, per), shell_ang_mom=np.zeros(S, dtype=np.int32),
                shell_prim_num=np.ones(S, dtype=np.int64), shell_prim_index=np.arange(S), shell_factor=np.ones(S),
                exponent=rng.uniform(0.3, 20.0, S), coefficient=np.ones(S), prim_factor=np.ones(S),
                ao_factor=np.ones(S), ao_num=S, mo_num=m, mo_coef=rng.standard_normal((m, S)))


def _molecules(call, form):
    if call == "mo_value" and form == pq.FORM_FP64:
        return [_chain(700, 10, 4), _chain(20, 10, 4)]   # 56 KB of shell lists, and 1.6 KB
    return [gen.config(1, walk_num=1), gen.config(0, walk_num=1)]


@pytest.mark.parametrize("call,form", [("mo_value", pq.FORM_FP64), ("mo_vgl", pq.FORM_MIXED),
                                       ("ao_hessian", pq.FORM_FP64)])
def test_threads_of_different_sizes(call, form):
    errors, wrong = [], []
    gate = threading.Barrier(4)

    def worker(d, seed):
        try:
            rng = np.random.default_rng(seed)
            xyz = np.asarray(d["nucl_coord"]).reshape(3, -1)
            pts = xyz.T[rng.integers(0, xyz.shape[1], P)] + rng.standard_normal((P, 3))
            c = torch.tensor(np.ascontiguousarray(pts.T), dtype=torch.float64, device="cuda")
            shape = {"mo_value": (P, d["mo_num"]), "mo_vgl": (P, 5, d["mo_num"]),
                     "ao_hessian": (3, P, 4, d["ao_num"])}[call]
            first, out = (torch.empty(shape, dtype=torch.float64, device="cuda") for _ in range(2))
            torch.cuda.synchronize()
            ctx = make_context(d, points=False, form=form)
            f = {"mo_value": pq.b200_mo_value_device, "mo_vgl": pq.b200_mo_vgl_device,
                 "ao_hessian": pq.b200_ao_hessian_device}[call]
            try:
                f(ctx, P, c.data_ptr(), first.data_ptr())
                pq.b200_synchronize(ctx)
                gate.wait(60)
                for _ in range(CALLS):
                    f(ctx, P, c.data_ptr(), out.data_ptr())
                pq.b200_synchronize(ctx)
                if not torch.equal(out, first):
                    wrong.append(d["ao_num"])
            finally:
                pq.context_destroy(ctx)
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))
            gate.abort()

    big, small = _molecules(call, form)
    torch.zeros(1, device="cuda")
    ts = [threading.Thread(target=worker, args=(d, i)) for i, d in enumerate([big, small, small, small])]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors and not wrong
