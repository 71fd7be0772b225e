"""Lanczos on several threads and streams at once: what each gets alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_threads_with_streams_of_their_own():
    import cytnx_b200 as c
    from cytnx_b200 import workloads as W

    ops = [W.build_two_site(W.xxz_spec(D), W.xxz_mpo_values(), seed=D, device=0) for D in (16, 33, 64, 101)]

    def solve(o, prec):
        H = c.TwoSiteHeff(*o[1:], o[0])
        return H.lanczos(o[0], maxiter=12, cvgcrit=1e-300, precision=prec)[0]

    alone = [[solve(o, p) for p in ("fp64", "bf16x3")] for o in ops]
    got = [[None, None] for _ in ops]
    errors = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3):
                    for k, p in enumerate(("fp64", "bf16x3")):
                        got[i][k] = solve(ops[i], p)
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()  # the operands are ready for every stream
    t = [threading.Thread(target=work, args=(i,)) for i in range(len(ops))]
    [x.start() for x in t]
    [x.join() for x in t]
    assert not errors and got == alone
