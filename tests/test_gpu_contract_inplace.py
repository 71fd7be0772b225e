"""Operands whose legs are in order but for legs of extent 1 are contracted in place: every order of
the legs of a U(1) tensor with one-state MPO and physical legs against the dense contraction."""
import itertools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tensor(c, bonds, labels, seed):
    u = c.UniTensor(bonds, labels=labels, rowrank=1, device=0)
    rng = np.random.default_rng(seed)
    u.flat_view().copy_(torch.from_numpy(rng.standard_normal(u.flat_view().numel())))
    return u


def _dense(u):
    return torch.from_numpy(u.contiguous().to_dense_numpy())


@pytest.mark.parametrize("degs", [(1, 1), (1, 2)])  # all MPO sectors of one state; one of two
def test_all_leg_orders(degs):
    import cytnx_b200 as c

    V = c.Bond(c.BD_KET, [[-1], [0], [1], [2]], [3, 1, 17, 5])
    w = c.Bond(c.BD_KET, [[0], [1]], list(degs))
    s = c.Bond(c.BD_KET, [[1], [-1]], [1, 1])
    T = _tensor(c, [w, V, s.redirect(), V.redirect()], ["w", "a", "s", "b"], 1)
    M = _tensor(c, [w.redirect(), w, s, s.redirect()], ["w", "v", "s", "t"], 2)
    E = _tensor(c, [w.redirect(), V.redirect(), V], ["w", "a", "x"], 3)
    for p in itertools.permutations(range(4)):
        Tp = T.permute(list(p))
        for other, eq, labels in ((M, "wasb,wvst->abvt", ["a", "b", "v", "t"]), (E, "wasb,wax->sbx", ["s", "b", "x"])):
            for q in itertools.permutations(range(other.rank())):
                got = _dense(c.Contract(Tp, other.permute(list(q))).permute(labels))
                ref = torch.einsum(eq, _dense(T), _dense(other))
                # sums of at most 46 products of N(0,1) values in FP64: n * eps relative to the norm
                assert torch.linalg.norm(got - ref) <= 46 * 2.3e-16 * torch.linalg.norm(ref)


def test_empty_legs_and_unit_blocks():
    """Blocks of a single element have no order at all; vectors are rows and columns at once."""
    import cytnx_b200 as c

    V = c.Bond(c.BD_KET, [[0], [1]], [1, 9])
    A = _tensor(c, [V, V.redirect()], ["i", "j"], 4)
    B = _tensor(c, [V, V.redirect()], ["j", "k"], 5)
    ref = _dense(A) @ _dense(B)
    for x, y in itertools.product((A, A.permute([1, 0])), (B, B.permute([1, 0]))):
        got = _dense(c.Contract(x, y).permute(["i", "k"]))
        assert torch.linalg.norm(got - ref) <= 9 * 2.3e-16 * torch.linalg.norm(ref)
