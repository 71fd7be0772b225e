"""Grouped FP64 products at the edges of their forms: scalar times vector, and tiles with
remainders in every direction, in all operand orientations, against torch in float64."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(tasks, ta, tb, seed=0):
    """tasks: list of (m, n, [k, ...]); operands and results packed back to back."""
    from cytnx_b200 import _lib

    class Task(ctypes.Structure):
        _fields_ = [("c_off", ctypes.c_int64), ("m", ctypes.c_int32), ("n", ctypes.c_int32), ("ldc", ctypes.c_int32),
                    ("pair_begin", ctypes.c_int32), ("pair_count", ctypes.c_int32), ("pad", ctypes.c_int32)]

    class Pair(ctypes.Structure):
        _fields_ = [("a_off", ctypes.c_int64), ("b_off", ctypes.c_int64), ("k", ctypes.c_int32), ("lda", ctypes.c_int32),
                    ("ldb", ctypes.c_int32), ("flags", ctypes.c_int32)]

    T, P, a, b, c = [], [], 1, 1, 1  # everything starts off a 16-byte boundary
    for m, n, ks in tasks:
        T.append(Task(c, m, n, n, len(P), len(ks), 0))
        c += m * n
        for k in ks:
            P.append(Pair(a, b, k, m if ta else max(k, 1), max(k, 1) if tb else n, int(ta) | 2 * int(tb)))
            a += m * k
            b += k * n
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    A, B = (torch.randn(x + 1, dtype=torch.float64, device="cuda", generator=g) for x in (a, b))
    C = torch.full((c + 1,), 7.0, dtype=torch.float64, device="cuda")
    lib, h = _lib.lib(), ctypes.c_void_p()
    _lib.check(lib.ctn_gemm_grouped_plan_create(len(T), (Task * len(T))(*T), len(P), (Pair * max(len(P), 1))(*P), ctypes.byref(h)))
    _lib.check(lib.ctn_gemm_grouped_f64(h, A.data_ptr(), B.data_ptr(), C.data_ptr(), _lib.stream_ptr()))
    torch.cuda.synchronize()
    lib.ctn_gemm_grouped_plan_destroy(h)
    assert float(C[0]) == 7.0 and float(C[-1]) == 7.0
    for t in T:
        ref = torch.zeros(t.m, t.n, dtype=torch.float64, device="cuda")
        mag = torch.zeros_like(ref)
        depth = 0
        for p in P[t.pair_begin: t.pair_begin + t.pair_count]:
            x = A[p.a_off: p.a_off + t.m * p.k].view(p.k, t.m).T if ta else A[p.a_off: p.a_off + t.m * p.k].view(t.m, p.k)
            y = B[p.b_off: p.b_off + p.k * t.n].view(t.n, p.k).T if tb else B[p.b_off: p.b_off + p.k * t.n].view(p.k, t.n)
            ref += x @ y
            mag += x.abs() @ y.abs()
            depth += p.k
        got = C[t.c_off: t.c_off + t.m * t.n].view(t.m, t.n)
        # each side's sum of `depth` products: at most depth * eps * sum |x||y| from the exact one
        assert bool(((got - ref).abs() <= 2 * max(depth, 1) * 1.2e-16 * mag).all())


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
def test_scalar_times_vector(ta, tb):
    # columns (n == 1, k == 1) and rows (m == 1, k == 1) around the 1024-element runs, empty sums,
    # pairs without k; A [m][1] and [1][m] are both contiguous, B likewise
    _run([(m, 1, [1] * c) for m, c in ((1, 1), (1023, 2), (1024, 1), (1025, 3), (5, 0), (4624, 4))] + [(7, 1, [1, 0, 1])], ta, tb)
    _run([(1, n, [1] * c) for n, c in ((1, 2), (1023, 1), (1025, 2), (300, 0))], ta, tb)


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
def test_tiles_with_remainders(ta, tb):
    sizes = [(1, 1, [3]), (31, 33, [16]), (32, 32, [15, 17]), (33, 31, [1, 0, 32]), (64, 32, [48]), (65, 97, [5, 7, 31]), (2, 70, []), (130, 3, [64])]
    _run(sizes, ta, tb)                               # small blocks: 32 x 32 tiles
    _run([(256, 256, [40]), (320, 288, [16, 33])], ta, tb)  # few tiles: 32 x 32 as well


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("m,n,ks", [(3000, 1000, [40, 7]),           # 64 x 32: 752 tiles of 64 x 64 are too few
                                    (2040, 2043, [40, 17]),          # 64 x 64, remainders in every direction
                                    (2048, 1985, [16, 3]),           # 64 x 64, two slices, one column in the last tile
                                    (2040, 2043, [9]),               # one slice: 1024 tiles are too few, 64 x 32
                                    (2945, 2999, [9]), (2945, 2999, [16])])  # 64 x 64 with one slice
def test_wide_tiles(m, n, ks, ta, tb):
    _run([(m, n, ks)], ta, tb)
