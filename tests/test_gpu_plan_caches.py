"""Contraction plans outlive a sweep of permutes over more layouts than a cache holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_permutes_do_not_push_out_contraction_plans():
    import cytnx_b200 as c
    from cytnx_b200 import unitensor as U

    def bond(n):
        return c.Bond(c.BD_KET, [[0], [1]], [n, 2])

    A = c.UniTensor([bond(3), bond(4).redirect()], labels=["a", "b"], rowrank=1, device=0)
    B = c.UniTensor([bond(4), bond(5).redirect()], labels=["b", "d"], rowrank=1, device=0)
    A._data.normal_(), B._data.normal_()
    before = set(U._PLANS)
    ref = c.Contract(A, B)
    mine = set(U._PLANS) - before
    assert len(mine) == 1
    for n in range(1, U._PERMUTES.cap + 20):
        t = c.UniTensor([bond(n), bond(3).redirect()], labels=["a", "b"], rowrank=1, device=0)
        t._data.normal_()
        p = t.permute([1, 0]).contiguous()
        if n % 100 == 1:  # and what the plan does is right
            assert torch.equal(p.permute([1, 0]).contiguous().flat_view(), t.flat_view())
    assert mine <= set(U._PLANS) and len(U._PERMUTES) <= U._PERMUTES.cap
    assert torch.equal(c.Contract(A, B).flat_view(), ref.flat_view())
