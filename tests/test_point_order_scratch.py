"""Scratch of the spatial point order (host logic, CPU only).

The batched loop and the chunked adjoint size the scratch for their largest
point count and then sort smaller counts in it, so its size must not fall as
the count grows, and it must hold what the sort lays out in it: 2-byte cell
codes, 2 KB of digit counts per block of the multi-block sort, 4-byte indices.
"""
import ctypes

import numpy as np

from qmckl_b200 import qmckl as pq


def _bytes():
    f = pq.lib()["_ZN2qb17point_order_bytesEl"]   # size_t qb::point_order_bytes(int64_t)
    f.restype, f.argtypes = ctypes.c_size_t, [ctypes.c_int64]
    return f


def _blocks(n):
    """Blocks of a pass: runs of 1024 to 4096 points, whole 256s, aiming at 64 blocks; whole 4096s for 592 blocks."""
    run = -(-min(4096, max(1024, -(-n // 64))) // 256) * 256
    if n > 592 * 4096:
        run = -(-(-(-n // 592)) // 4096) * 4096
    return -(-n // run)


def test_scratch_serves_every_smaller_count():
    f = _bytes()
    edges = np.arange(256, 400_000, 256)
    counts = sorted(set(int(e + o) for e in edges for o in (-1, 0, 1)) | {66_000, 65_000, 1_000_000, 2_424_832, 2_424_833, 6_170_000})
    size = [f(n) for n in counts]
    assert all(a <= b for a, b in zip(size, size[1:]))


def test_scratch_holds_the_layout():
    f = _bytes()
    for n in [4097, 16_385, 65_535, 65_536, 65_537, 131_073, 262_144, 262_145, 1_000_001, 2_424_832, 2_424_833, 6_170_000]:
        codes = -(-2 * n // 256) * 256
        assert f(n) >= codes + 2048 * _blocks(n) + 4 * n
    assert f(4096) == 0
