"""The fused step of the plain Lanczos recurrence at the sizes and alignments that select its branches."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def recurrence(d, v, steps):
    """The plain recurrence for the operator diag(d) in FP64 numpy (Lanczos_Gnd.cpp)."""
    q, alpha, beta = [v / np.linalg.norm(v)], [], []
    for i in range(steps):
        w = d * q[i]
        alpha.append(w @ q[i])
        w = w - alpha[i] * q[i] - (beta[i - 1] * q[i - 1] if i else 0.0)
        beta.append(np.linalg.norm(w))
        q.append(w / beta[i])
    return np.array(q), np.array(alpha), np.array(beta)


# odd n: every other Krylov vector starts off a 16-byte boundary; `shift` moves the matvec's result;
# 300007 takes several rounds of the capped grid, 255 and below less than one CTA
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [4, 5, 255, 512, 1023, 1025, 300006, 300007])
def test_krylov_vectors_match_the_recurrence(n, shift):
    from cytnx_b200 import _lib

    maxiter = 3
    rng = np.random.default_rng(n)
    d, v = rng.uniform(1.0, 2.0, n), rng.standard_normal(n)
    dt, v0 = torch.from_numpy(d).cuda(), torch.from_numpy(v).cuda()
    kry = torch.zeros((maxiter + 1) * n, dtype=torch.float64, device="cuda")
    work = torch.empty(max(4 * n + 64, n + 1104 + maxiter) + shift, dtype=torch.float64, device="cuda")[shift:]
    eig = torch.empty(n, dtype=torch.float64, device="cuda")

    def mv(user, x, y, stream):
        at = (x - kry.data_ptr()) // 8
        torch.mul(dt, kry[at:at + n], out=work[:n])
        return 0

    fn = _lib.MATVEC_FN(mv)
    e, it = ctypes.c_double(), ctypes.c_int()
    _lib.check(_lib.lib().ctn_lanczos_gnd(fn, None, v0.data_ptr(), n, maxiter, 1e-300, kry.data_ptr(),
                                          work.data_ptr(), eig.data_ptr(), ctypes.byref(e), ctypes.byref(it), _lib.stream_ptr()),
               "lanczos")
    q, alpha, beta = recurrence(d, v, maxiter)
    assert it.value == maxiter
    # rounding of a step (sums of n terms in log2(n) + n / 2^18 levels or better: below 64 eps) grows by at
    # most (|d| + alpha + beta) / beta < 5 / beta per step
    tol = 64 * np.finfo(float).eps * np.prod(5.0 / beta)
    assert np.abs(kry.cpu().numpy().reshape(maxiter + 1, n) - q).max() <= tol
    t = np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1)
    assert abs(e.value - np.linalg.eigvalsh(t)[0]) <= tol


def test_breakdown_of_an_eigenvector():
    """beta == 0 in the first step: one iteration, the next vector is zeros."""
    from cytnx_b200 import _lib

    n, maxiter = 6, 4
    kry = torch.ones((maxiter + 1) * n, dtype=torch.float64, device="cuda")
    work = torch.empty(n + 1104 + maxiter, dtype=torch.float64, device="cuda")
    v0, eig = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    v0[2] = 3.0

    def mv(user, x, y, stream):
        at = (x - kry.data_ptr()) // 8
        torch.mul(kry[at:at + n], 1.5, out=work[:n])
        return 0

    fn = _lib.MATVEC_FN(mv)
    e, it = ctypes.c_double(), ctypes.c_int()
    _lib.check(_lib.lib().ctn_lanczos_gnd(fn, None, v0.data_ptr(), n, maxiter, 1e-300, kry.data_ptr(),
                                          work.data_ptr(), eig.data_ptr(), ctypes.byref(e), ctypes.byref(it), _lib.stream_ptr()),
               "lanczos")
    assert it.value == 1 and e.value == 1.5
    assert torch.equal(kry[n:2 * n], torch.zeros_like(v0)) and torch.equal(eig, v0 / 3.0)
