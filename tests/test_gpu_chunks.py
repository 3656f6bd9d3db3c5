"""Evaluations in several chunks of points (GPU): the FP64 MO VGL and value
and the adjoint of both forms, with their scratch bound to a few tiles, against
the same call in one chunk and the oracle.  Chunk counts with a last chunk that
is shorter than the others, down to one tile or a part of one, and with one
that is not.

A chunk changes no sum of the forward, which is therefore the same to the last
bit; the FP64 adjoint sums dL/dC and dL/dR in another order (1e-13 of the
largest entry).  A chunk of the mixed adjoint is compared with the call of its
points alone.
"""
import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from qmckl_b200 import gen
from qmckl_b200 import qmckl as pq
from qmckl_b200.system import make_context

pytestmark = pytest.mark.gpu


def _case(P, m):
    d = gen.config(0, walk_num=1)
    rng = np.random.default_rng(P + m)
    d["mo_coef"] = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((d["ao_num"], m)))[0].T)
    d["mo_num"] = m
    xyz = np.asarray(d["nucl_coord"]).reshape(3, -1).T
    return d, xyz[rng.integers(0, xyz.shape[0], P)] + rng.standard_normal((P, 3)), rng.standard_normal((P, 5, m))


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


# limits: bytes of about 1, 3 and 4 of the tiles of 32 points of a 90-AO molecule
@pytest.mark.parametrize("P", [33, 300, 301, 321])
@pytest.mark.parametrize("comps,m", [(5, 90), (5, 31), (1, 33)])
@pytest.mark.parametrize("tiles", [1, 3, 4])
def test_forward_in_chunks(P, comps, m, tiles):
    d, pts, _ = _case(P, m)
    c = _dev(pts.T)
    f = pq.b200_mo_vgl_device if comps == 5 else pq.b200_mo_value_device
    one, many = (torch.full((P, comps, m), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        f(ctx, P, c.data_ptr(), one.data_ptr())
        n0 = pq.b200_kernel_launch_count()
        pq.b200_set_scratch_limit(ctx, tiles * 8 * (32 * comps + 6) * d["ao_num"])
        f(ctx, P, c.data_ptr(), many.data_ptr())
        launches = pq.b200_kernel_launch_count() - n0
        pq.b200_synchronize(ctx)
    finally:
        pq.context_destroy(ctx)
    chunks = -(-(-(-P // 32)) // tiles)
    assert launches == 1 + 2 * chunks   # the point order, AOs and contraction of each chunk
    assert torch.equal(one, many)


CASES = [(300, 90, 100), (301, 31, 64), (257, 64, 64), (130, 33, 64), (1000, 20, 333)]   # P, MOs, points per chunk


def _adjoint(ctx, pts, w, shapes, outputs):
    out = [torch.full(s, float("nan"), dtype=torch.float64, device="cuda") for s in shapes]
    c, dw = _dev(pts.T), _dev(w)
    torch.cuda.synchronize()
    n0 = pq.b200_kernel_launch_count()
    pq.b200_mo_vgl_adjoint_device(ctx, pts.shape[0], c.data_ptr(), dw.data_ptr(),
                                  *(o.data_ptr() if k in outputs else 0 for k, o in zip("cnr", out)))
    launches = pq.b200_kernel_launch_count() - n0
    pq.b200_synchronize(ctx)
    return out, launches


@pytest.mark.parametrize("P,m,points_per_chunk", CASES)
@pytest.mark.parametrize("outputs", ["cnr", "c", "n", "r"])
def test_adjoint_in_chunks_fp64(P, m, points_per_chunk, outputs):
    d, pts, w = _case(P, m)
    A, N = d["ao_num"], d["nucl_num"]
    # bytes per point: AO tile, weights and dL/dC products
    per_point = (8 * 164 * A + 8 * 160 * m + 8 * A * m + 20 * A) // 32
    ctx = make_context(d, points=False, form=pq.FORM_FP64)
    try:
        one, n_one = _adjoint(ctx, pts, w, ((m, A), (N, 3), (3, P)), outputs)
        pq.b200_set_scratch_limit(ctx, points_per_chunk * per_point)
        many, n_many = _adjoint(ctx, pts, w, ((m, A), (N, 3), (3, P)), outputs)
    finally:
        pq.context_destroy(ctx)
    assert n_many > n_one
    ref = O.mo_vgl_adjoint(O.Basis(d), pts, d["nucl_coord"], d["mo_coef"], w)
    for k, a, b, r in zip("cnr", one, many, ref):
        if k in outputs:
            r = r.T if k == "r" else r
            assert float((a - b).abs().max()) <= 1e-13 * float(a.abs().max())
            assert np.abs(b.cpu().numpy() - r).max() <= 1e-10 * np.abs(r).max()


@pytest.mark.parametrize("P,m,points_per_chunk", CASES)
@pytest.mark.parametrize("outputs", ["cnr", "c", "n", "r"])
def test_adjoint_in_chunks_mixed(P, m, points_per_chunk, outputs):
    """A chunk of the mixed adjoint is the call of its points alone: dL/dr the same bits, dL/dC the chunks' sum."""
    d, pts, w = _case(P, m)
    A, N = d["ao_num"], d["nucl_num"]
    chunks = -(-P // points_per_chunk)
    step = -(-P // chunks)
    ctx = make_context(d, points=False, form=pq.FORM_MIXED)
    try:
        parts = [_adjoint(ctx, pts[a:a + step], w[a:a + step], ((m, A), (N, 3), (3, min(step, P - a))), outputs)[0]
                 for a in range(0, P, step)]
        n_one = _adjoint(ctx, pts, w, ((m, A), (N, 3), (3, P)), outputs)[1]
        pq.b200_set_scratch_limit(ctx, points_per_chunk * 30 * ((A + 7) // 8 * 8))   # the chunk's AO pieces
        many, n_many = _adjoint(ctx, pts, w, ((m, A), (N, 3), (3, P)), outputs)
    finally:
        pq.context_destroy(ctx)
    assert n_many > n_one
    want = [parts[0][0].clone(), parts[0][1].clone(), torch.cat([p[2] for p in parts], 1)]
    for p in parts[1:]:
        want[0] += p[0]
        want[1] += p[1]
    if "c" in outputs:
        assert torch.equal(many[0], want[0])
    if "n" in outputs:
        assert float((many[1] - want[1]).abs().max()) <= 1e-13 * float(want[1].abs().max())
    if "r" in outputs:
        assert torch.equal(many[2], want[2])


def test_adjoint_last_chunk_is_the_smaller_one():
    """131,073 points of 1000 AOs, the mixed adjoint as a context's first call: chunks of 65,537 and 65,536 points,
    whose sorts take 52 and 64 blocks in the scratch made for the first."""
    rng = np.random.default_rng(5)
    charges = [6.0] * 20 + [1.0] * 20
    xyz = gen.place_nuclei(rng, 40, 15.9)
    m, P = 8, 131_073
    d = gen.build_system(rng, charges, xyz, gen.SHAPES["tz_heavy"], gen.SHAPES["tz_h"], m, 1, elec_num=2)
    pts = xyz[rng.integers(0, 40, P)] + rng.standard_normal((P, 3))
    c, w = _dev(pts.T), _dev(rng.standard_normal((P, 5, m)))
    res = []
    for form in (pq.FORM_MIXED, pq.FORM_FP64):
        out = [torch.full(s, float("nan"), dtype=torch.float64, device="cuda")
               for s in ((m, d["ao_num"]), (d["nucl_num"], 3), (3, P))]
        torch.cuda.synchronize()
        ctx = make_context(d, points=False, form=form)
        try:
            pq.b200_mo_vgl_adjoint_device(ctx, P, c.data_ptr(), w.data_ptr(), *(o.data_ptr() for o in out))
            pq.b200_synchronize(ctx)
        finally:
            pq.context_destroy(ctx)
        res.append(out)
    assert d["ao_num"] == 1000
    for a, b in zip(*res):
        assert float((a - b).abs().max()) <= 1e-6 * float(b.abs().max())
