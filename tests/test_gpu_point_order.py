"""The spatial point order itself (GPU): the permutation is the stable sort by
the Morton codes of 32^3 cells, at the edges of its forms (one block up to 4096
points; runs of 1024 to 4096 points on up to 592 blocks; several runs per block
beyond 2,424,832), with scratch made for that count, or for a larger one, and
nothing written past it."""
import ctypes

import numpy as np
import pytest
import torch

from qmckl_b200 import qmckl as pq

pytestmark = pytest.mark.gpu

LO, HI = np.array([-5.0, -4.0, -7.0]), np.array([6.0, 41.0, 8.0])
GUARD = 4096


def _spread(x):
    return sum(((x >> b) & 1) << (3 * b) for b in range(5))


def _reference(pts):
    inv = 1.0 / max(1.0, (HI - LO).max() / 32.0)
    cell = np.clip(np.floor((pts - LO) * inv), 0, 31).astype(np.int64)
    key = _spread(cell[:, 0]) | (_spread(cell[:, 1]) << 1) | (_spread(cell[:, 2]) << 2)
    return np.argsort(key, kind="stable")


@pytest.mark.parametrize("P,room", [(1, 1), (33, 33), (4096, 4096), (4097, 4097), (10_001, 10_001), (65_536, 65_537),
                                    (65_537, 65_537), (65_000, 66_000), (262_145, 262_145), (2_424_832, 2_424_832),
                                    (2_424_833, 2_424_833), (3_000_001, 3_100_000)])
def test_point_order(P, room):
    lib = pq.lib()
    size = lib["_ZN2qb17point_order_bytesEl"]
    size.restype, size.argtypes = ctypes.c_size_t, [ctypes.c_int64]
    order = lib["_ZN2qb11point_orderEPKdlS1_S1_PvPiP11CUstream_stl"]
    order.restype = ctypes.c_int
    order.argtypes = [ctypes.c_void_p, ctypes.c_int64] + [ctypes.c_void_p] * 5 + [ctypes.c_int64]
    rng = np.random.default_rng(P)
    pts = rng.uniform(LO - 2.0, HI + 2.0, (P, 3))
    pts[: P // 2] = pts[0] + 0.3 * rng.standard_normal((P // 2, 3))   # half of them in a few cells
    c = torch.tensor(np.ascontiguousarray(pts.T), device="cuda")
    n = size(room)
    scratch = torch.full((n + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    perm = torch.full((P + 64,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.current_stream().cuda_stream
    assert order(c.data_ptr(), P, LO.ctypes.data, HI.ctypes.data, scratch.data_ptr(), perm.data_ptr(), s, P) == 0
    torch.cuda.synchronize()
    assert np.array_equal(perm[:P].cpu().numpy(), _reference(pts))
    assert bool((perm[P:] == -7).all()) and bool((scratch[n:] == 0xA5).all())
