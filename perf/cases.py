"""The work that a DMRG or TEBD program has this package do, as cases to be timed.

Every case goes through the public entry points (``Tensor`` / ``UniTensor`` permute + contiguous,
``Network.Launch``, ``TwoSiteHeff``, ``BatchedTwoSiteHeff``, ``env.left_update`` /
``right_update``, ``U1MPS.energy`` with its gradient).  The block structures are those of the
package's own configurations: the spin-1/2 XXZ chain with U(1) sectors ~ exp(-q^2/72), and the
spinful Hubbard chain with (N, 2Sz) sectors of Gaussian weight.  Values are ~N(0,1) in the
symmetry-allowed blocks, environments Hermitian, wavefunctions normalised.

``exact`` computes the same results from dense tensors with torch in float64; it shares only the
sector sizes and the MPO's entries (inputs, not results) with the package.
"""
import functools
import math

import numpy as np
import torch

import cytnx_b200 as cytnx
from cytnx_b200 import env, workloads
from cytnx_b200.autodiff import U1MPS, mps_bond_sectors

KET, BRA = 1, -1  # sign of a leg's charge in the flux rule (ket +q, bra -q)

DTYPES = {"float64": torch.float64, "float32": torch.float32, "complex128": torch.complex128,
          "complex64": torch.complex64, "int64": torch.int64, "int32": torch.int32, "int16": torch.int16,
          "bool": torch.bool}
BATCH_ALIGN = 32  # the batch places every problem's vector on a multiple of this many elements


# ---------------------------------------------------------------- cases
def listed():
    return [
        # materialising a lazy permutation of a small site tensor: what a script does between
        # contractions, bound by the call and one launch
        {"name": "permute_small_f64", "kind": "permute", "shape": "64,2,2,64", "mapper": "3,1,2,0", "dtype": "float64"},
        # a two-site tensor of a large dense bond dimension, reversed: bound by memory
        {"name": "permute_large_f32", "kind": "permute", "shape": "4096,3,3,4096", "mapper": "3,1,2,0",
         "dtype": "float32"},
        # a ragged tensor of a narrow type: no extent is a multiple of a vector or a tile
        {"name": "permute_ragged_i16", "kind": "permute", "shape": "1021,3,37,509", "mapper": "3,1,0,2",
         "dtype": "int16"},
        # every block of a U(1) wavefunction permuted and put into the order of its new legs
        {"name": "blocks_xxz_D1024", "kind": "blocks", "model": "xxz", "D": 1024, "mapper": "3,0,2,1"},
        # single-site matvec of plain dense DMRG through Network: small calls, one after another
        {"name": "dense_site_D64", "kind": "dense_site", "D": 64},
        # two-site effective Hamiltonian, FP64: a small odd bond dimension at the chain's ends ...
        {"name": "heff_fp64_D301", "kind": "heff", "D": 301, "precision": "fp64"},
        # ... and the largest
        {"name": "heff_fp64_D4096", "kind": "heff", "D": 4096, "precision": "fp64"},
        # the same operator in split precision, the tiles as a program gets them without tuning
        {"name": "heff_bf16x3_D4096", "kind": "heff", "D": 4096, "precision": "bf16x3"},
        # many uneven Hubbard problems in one batch
        {"name": "batch_3xtf32_32", "kind": "batch", "n": 32, "dmin": 128, "dmax": 2048, "dseed": 0,
         "precision": "3xtf32"},
        # the environment update after a DMRG step
        {"name": "env_left_D1024", "kind": "env", "D": 1024, "side": "left"},
        # energy of an MPS and its gradient: contractions forward and backward
        {"name": "mps_gradient_L16_D192", "kind": "mps", "L": 16, "D": 192},
        # ground-state Lanczos as a DMRG step runs it
        {"name": "lanczos_fp64_D1024", "kind": "lanczos", "D": 1024, "iters": 20, "precision": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["permute", "permute", "blocks", "dense_site", "heff", "heff", "batch", "env", "mps", "lanczos"])
    prec = rng.choice(["fp64", "bf16x3", "3xtf32"])
    if kind == "permute":
        dtype = rng.choice(sorted(DTYPES))
        es = torch.empty(0, dtype=DTYPES[dtype]).element_size()
        rank = rng.randint(2, 5)
        n = _log(rng, 1 << 10, (1 << 29) // es)
        share = [rng.uniform(0.05, 1.0) for _ in range(rank)]
        shape = [max(1, int(n ** (s / sum(share)))) for s in share]
        mapper = list(range(rank))
        while mapper == list(range(rank)):
            rng.shuffle(mapper)
        return {"kind": kind, "shape": ",".join(map(str, shape)), "mapper": ",".join(map(str, mapper)), "dtype": dtype}
    if kind == "blocks":
        model = rng.choice(["xxz", "hubbard"])
        mapper = [0, 1, 2, 3]
        while mapper == [0, 1, 2, 3]:
            rng.shuffle(mapper)
        return {"kind": kind, "model": model, "D": _log(rng, 32, 4096 if model == "xxz" else 1024),
                "mapper": ",".join(map(str, mapper))}
    if kind == "dense_site":
        return {"kind": kind, "D": _log(rng, 12, 256)}
    if kind == "heff":
        return {"kind": kind, "D": _log(rng, 32, 4096), "precision": prec}
    if kind == "batch":
        dmax = _log(rng, 96, 2048)
        return {"kind": kind, "n": rng.randint(1, min(24, int(9 * (2048 / dmax) ** 2))), "dmin": rng.randint(32, dmax // 2),
                "dmax": dmax, "dseed": rng.randint(1, 10 ** 6), "precision": rng.choice(["bf16x3", "3xtf32"])}
    if kind == "env":
        return {"kind": kind, "D": _log(rng, 32, 1024), "side": rng.choice(["left", "right"])}
    if kind == "mps":
        return {"kind": kind, "L": rng.randrange(6, 17, 2), "D": _log(rng, 8, 192)}
    return {"kind": kind, "D": _log(rng, 32, 1024), "iters": rng.randint(4, 20), "precision": prec}


# ---------------------------------------------------------------- block structures
class Legs:
    """Legs (sign, charges, degeneracies) of a block-sparse tensor and its blocks, in the order
    of their charge indices with the last leg fastest."""

    def __init__(self, *legs):
        self.legs = [(s, np.asarray(q, dtype=np.int64).reshape(len(d), -1), np.asarray(d, dtype=np.int64))
                     for s, q, d in legs]
        idx, tot = np.zeros((1, 0), dtype=np.int64), np.zeros((1, self.legs[0][1].shape[1]), dtype=np.int64)
        for s, q, d in self.legs:
            n = len(d)
            idx = np.concatenate([np.repeat(idx, n, axis=0), np.tile(np.arange(n), len(idx))[:, None]], axis=1)
            tot = np.repeat(tot, n, axis=0) + s * np.tile(q, (len(tot), 1))
        self.itoi = idx[(tot == 0).all(axis=1)]
        self.shapes = np.stack([d[self.itoi[:, i]] for i, (_, _, d) in enumerate(self.legs)], axis=1)
        self.sizes = self.shapes.prod(axis=1)
        self.offs = np.concatenate([[0], np.cumsum(self.sizes)])
        self.nelem = int(self.offs[-1])
        self.dims = [int(d.sum()) for _, _, d in self.legs]

    def bonds(self):
        return [cytnx.Bond(cytnx.BD_KET if s == KET else cytnx.BD_BRA, q, d) for s, q, d in self.legs]

    def permuted(self, mapper):
        return Legs(*[self.legs[i] for i in mapper])

    def _slices(self):
        start = [np.concatenate([[0], np.cumsum(d)]) for _, _, d in self.legs]
        for b, t in enumerate(self.itoi.tolist()):
            yield b, tuple(slice(int(start[i][q]), int(start[i][q + 1])) for i, q in enumerate(t))

    def dense(self, flat):
        full = torch.zeros(self.dims, dtype=flat.dtype, device=flat.device)
        for b, sl in self._slices():
            full[sl] = flat[self.offs[b]: self.offs[b + 1]].view(*self.shapes[b].tolist())
        return full

    def flat(self, full):
        out = torch.empty(self.nelem, dtype=full.dtype, device=full.device)
        for b, sl in self._slices():
            out[self.offs[b]: self.offs[b + 1]] = full[sl].reshape(-1)
        return out


class TwoSite:
    """Structure of a two-site problem: psi[a,s1,s2,b], L[w,a,a'], M[w,w',s,s'], R[w,b,b']."""

    def __init__(self, model, D):
        if model == "xxz":
            ql, dl = qr, dr = workloads.u1_sector_sizes(D)
            phys, inner, self.conj = workloads.SPIN_PHYS_Q, workloads.XXZ_INNER_Q, workloads.XXZ_P
            self.mpo = workloads.xxz_mpo_values(1.0, 1.0, 0.0)
        else:
            ql, dl = workloads.hubbard_sector_sizes(D, 4.0, (0, 0))
            qr, dr = workloads.hubbard_sector_sizes(D, 4.0, (-2, 0))
            phys, inner, self.conj = workloads.HUB_PHYS_Q, workloads.HUB_INNER_Q, workloads.HUB_P
            self.mpo = workloads.hubbard_mpo_values(4.0, 1.0)
        s, w = (phys, [1] * len(phys)), (inner, [1] * len(inner))
        self.psi = Legs((KET, ql, dl), (BRA, *s), (BRA, *s), (BRA, qr, dr))
        self.L = Legs((BRA, *w), (BRA, ql, dl), (KET, ql, dl))
        self.R = Legs((KET, *w), (KET, qr, dr), (BRA, qr, dr))
        self.M = Legs((KET, *w), (BRA, *w), (KET, *s), (BRA, *s))
        self.A = Legs((KET, ql, dl), (BRA, *s), (BRA, qr, dr))  # a single site between the bonds

    def mpo_dense(self):
        m = np.zeros(self.M.dims)
        for key, v in self.mpo.items():
            m[key] = v
        return torch.from_numpy(m)

    def environment(self, legs, rng, dtype=np.float64):
        """~N(0,1) with X[w,a,a'] = X[conj(w),a',a]."""
        x = rng.standard_normal(legs.nelem)
        at = {tuple(t): b for b, t in enumerate(legs.itoi.tolist())}
        out = np.empty_like(x)
        for (w, p, q), b in at.items():
            c = at[(self.conj[w], q, p)]
            one, two = (x[legs.offs[k]: legs.offs[k + 1]].reshape(legs.shapes[k][1:]) for k in (b, c))
            out[legs.offs[b]: legs.offs[b + 1]] = (0.5 * (one + two.T)).reshape(-1)
        return out.astype(dtype)

    def vector(self, legs, rng, dtype=np.float64):
        x = rng.standard_normal(legs.nelem)
        return (x / np.linalg.norm(x)).astype(dtype)

    @functools.lru_cache(maxsize=None)
    def matvec_flops(self):
        """2 m n k over the block pairs of L psi and X3 R whose results an entry of the folded
        MPO reads or writes, and of the fold itself."""
        m = self.mpo_dense().numpy() != 0
        fold = np.einsum("wvsx,vuty->wstuxy", m.astype(float), m.astype(float)) != 0
        reads, writes = fold.any(axis=(3, 4, 5)), fold.any(axis=(0, 1, 2))
        mults = float(fold.sum()) / max(1, writes.sum())
        lby, rby = {}, {}
        for (w, a, x), s in zip(self.L.itoi.tolist(), self.L.shapes.tolist()):
            lby.setdefault(a, []).append((w, s[2]))
        for (u, b, y), s in zip(self.R.itoi.tolist(), self.R.shapes.tolist()):
            rby.setdefault(y, []).append((u, s[1]))
        f = 0.0
        for (a, s, t, b), sh in zip(self.psi.itoi.tolist(), self.psi.shapes.tolist()):
            f += sum(2.0 * sh[0] * x * sh[3] for w, x in lby.get(a, ()) if reads[w, s, t])
            f += sum(2.0 * sh[0] * k * sh[3] + 2.0 * mults * sh[0] * k for u, k in rby.get(b, ()) if writes[u, s, t])
        return float(f)

    @functools.lru_cache(maxsize=None)
    def env_flops(self, side):
        """The two large contractions of an environment update (with A and with its adjoint)."""
        legs, bond = (self.L, 0) if side == "left" else (self.R, 2)
        by = {}
        for (w, p, q), s in zip(legs.itoi.tolist(), legs.shapes.tolist()):
            by.setdefault(p, []).append(s[2])
        f = 0.0
        for t, sh in zip(self.A.itoi.tolist(), self.A.shapes.tolist()):
            f += sum(4.0 * sh[0] * x * sh[2] for x in by.get(t[bond], ()))
        return float(f)


@functools.lru_cache(maxsize=None)
def two_site(model, D):
    return TwoSite(model, D)


@functools.lru_cache(maxsize=None)
def mps_legs(L, D):
    """(site legs, boundary dimension of each site's left bond) of a total-Sz = 0 MPS."""
    bonds = [mps_bond_sectors(L, k, D) for k in range(L + 1)]
    s = (workloads.SPIN_PHYS_Q, [1, 1])
    return [Legs((KET, *bonds[k]), (BRA, *s), (BRA, *bonds[k + 1])) for k in range(L)]


def batch_dims(case):
    return workloads.hubbard_batch_dims(case["n"], case["dmin"], case["dmax"], case["dseed"])


# ---------------------------------------------------------------- inputs (from the seed alone)
def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _ints(text):
    return [int(t) for t in text.split(",")]


def _permute_input(case, seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    shape, dt = _ints(case["shape"]), DTYPES[case["dtype"]]
    if dt.is_floating_point or dt.is_complex:
        return torch.randn(shape, dtype=dt, device=_device(), generator=g)
    if dt == torch.bool:
        return torch.randint(0, 2, shape, dtype=torch.uint8, device=_device(), generator=g).to(dt)
    return torch.randint(-30000, 30000, shape, dtype=dt, device=_device(), generator=g)


def _dense_site_input(case, seed):
    rng, D = np.random.default_rng(seed), case["D"]
    L, R = (rng.standard_normal((D, 5, D)) for _ in range(2))
    L, R = (0.5 * (x + x.transpose(2, 1, 0)) for x in (L, R))
    W = np.zeros((5, 5, 2, 2))
    for key, v in workloads.xxz_mpo_values(1.0, 1.0, 0.0).items():
        W[key] = v
    A = rng.standard_normal((D, 2, D))
    return [torch.from_numpy(x).to(_device()) for x in (L, W, R, A / np.linalg.norm(A))]


def _two_site_input(case, seed):
    """Flat (psi, L, R) of the XXZ problem."""
    p, rng = two_site("xxz", case["D"]), np.random.default_rng(seed)
    flats = p.vector(p.psi, rng), p.environment(p.L, rng), p.environment(p.R, rng)
    return [torch.from_numpy(x).to(_device()) for x in flats]


def _env_input(case, seed):
    p, rng = two_site("xxz", case["D"]), np.random.default_rng(seed)
    X = p.environment(p.L if case["side"] == "left" else p.R, rng)
    A = rng.standard_normal(p.A.nelem) / math.sqrt(2.0 * case["D"])
    return [torch.from_numpy(x).to(_device()) for x in (X, A)]


def _batch_input(case, seed):
    """(psi, L, R) flats of every problem, FP32."""
    out = []
    for i, D in enumerate(batch_dims(case)):
        p, rng = two_site("hubbard", D), np.random.default_rng([seed, i])
        out.append((p.vector(p.psi, rng, np.float32), p.environment(p.L, rng, np.float32),
                    p.environment(p.R, rng, np.float32)))
    return out


def _mps_input(case, seed):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy(rng.standard_normal(s.nelem) / math.sqrt(2.0 * s.dims[0])).to(_device())
            for s in mps_legs(case["L"], case["D"])]


# ---------------------------------------------------------------- prepare and run
def _block(legs, labels, rowrank, flat):
    u = cytnx.UniTensor(legs.bonds(), labels=labels, rowrank=rowrank, device=0)
    u.flat_view().copy_(flat)
    return u


def _mpo(p):
    u = cytnx.UniTensor(p.M.bonds(), labels=["w0", "w1", "s", "sp"], rowrank=2, device=0)
    u.flat_view().copy_(p.M.flat(p.mpo_dense()))
    return u


class _OneSite(cytnx.LinOp):
    """Single-site H_eff as a DMRG script writes it: a Network with the environments put once."""

    def __init__(self, L, W, R, n):
        super().__init__("mv", n, cytnx.Type.Double, cytnx.Device.cuda)
        self.net = cytnx.Network()
        self.net.FromString(["A: a,s,b", "L: a,w,ap", "W: w,w2,s,sp", "R: b,w2,bp", "TOUT: ap,sp,bp"])
        self.net.PutUniTensors(["L", "W", "R"], [L, W, R])

    def matvec(self, v):
        self.net.PutUniTensor("A", v)
        out = self.net.Launch()
        out.relabel_(v.labels())
        return out


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "permute":
        state["t"] = cytnx.Tensor.from_torch(_permute_input(case, seed))
        state["mapper"] = _ints(case["mapper"])
    elif kind == "blocks":
        p = two_site(case["model"], case["D"])
        x = torch.from_numpy(p.vector(p.psi, np.random.default_rng(seed)))
        state["u"] = _block(p.psi, ["a", "s1", "s2", "b"], 1, x)
        state["mapper"] = _ints(case["mapper"])
    elif kind == "dense_site":
        L, W, R, A = (cytnx.Tensor.from_torch(x) for x in _dense_site_input(case, seed))
        Lu, Wu = cytnx.UniTensor(L, False, -1, ["a", "w", "ap"]), cytnx.UniTensor(W, False, -1, ["w", "w2", "s", "sp"])
        Ru, Au = cytnx.UniTensor(R, False, -1, ["b", "w2", "bp"]), cytnx.UniTensor(A, False, -1, ["a", "s", "b"])
        state["H"], state["v"] = _OneSite(Lu, Wu, Ru, 2 * case["D"] ** 2), Au
    elif kind in ("heff", "lanczos"):
        p = two_site("xxz", case["D"])
        x, l, r = _two_site_input(case, seed)
        psi = _block(p.psi, ["a", "s1", "s2", "b"], 1, x)
        L, R, M = _block(p.L, ["w", "a", "ap"], 1, l), _block(p.R, ["w", "b", "bp"], 1, r), _mpo(p)
        state["H"] = cytnx.TwoSiteHeff(L, M, M.clone(), R, psi, precision=case["precision"])
        state["H"].bind()
        state["psi"] = psi
    elif kind == "batch":
        dims, data = batch_dims(case), _batch_input(case, seed)
        B = cytnx.BatchedTwoSiteHeff(workloads.hubbard_batch(dims), precision=case["precision"])
        B.set_env(B.gather([d[1] for d in data], "L"), B.gather([d[2] for d in data], "R"))
        state["B"], state["psi"] = B, B.gather([d[0] for d in data], "psi")
    elif kind == "env":
        p = two_site("xxz", case["D"])
        X, A = _env_input(case, seed)
        left = case["side"] == "left"
        state["X"] = _block(p.L if left else p.R, ["w", "a", "ap"], 1, X)
        state["A"], state["M"] = _block(p.A, ["a", "s", "b"], 2, A), _mpo(p)
        state["update"] = env.left_update if left else env.right_update
    elif kind == "mps":
        m = U1MPS(case["L"], case["D"], seed=0)
        with torch.no_grad():
            for q, x in zip(m.params, _mps_input(case, seed)):
                q.copy_(x)
        state["mps"] = m
    else:
        raise ValueError(f"unknown kind {kind}")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "permute":
        return state["t"].permute(state["mapper"]).contiguous().to_torch()
    if kind == "blocks":
        return state["u"].permute(state["mapper"]).contiguous().flat_view()
    if kind == "dense_site":
        return state["H"].matvec(state["v"]).get_block_().to_torch()
    if kind == "heff":
        return state["H"].matvec(state["psi"]).flat_view()
    if kind == "lanczos":
        E, vec, _ = state["H"].lanczos(state["psi"], maxiter=case["iters"], cvgcrit=1e-300)
        return {"energy": E, "vector": vec.flat_view()}
    if kind == "batch":
        return state["B"].matvec(state["psi"])
    if kind == "env":
        return state["update"](state["X"], state["A"], state["M"]).contiguous().flat_view()
    E = state["mps"].energy()
    return {"energy": E.detach(), "gradient": list(torch.autograd.grad(E, state["mps"].params))}


# ---------------------------------------------------------------- accounting
def work(case):
    kind = case["kind"]
    if kind == "permute":
        n = math.prod(_ints(case["shape"]))
        return {"bytes": 2.0 * n * torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size(), "flops": 0.0}
    if kind == "blocks":
        return {"bytes": 16.0 * two_site(case["model"], case["D"]).psi.nelem, "flops": 0.0}
    if kind == "dense_site":
        D = case["D"]
        return {"bytes": 8.0 * (2 * 5 * D * D + 100 + 2 * 2 * D * D), "flops": 2.0 * 2 * (5 * 2 * D ** 3)}
    if kind in ("heff", "lanczos"):
        p, reps = two_site("xxz", case["D"]), case.get("iters", 1)
        return {"bytes": 8.0 * (2 * p.psi.nelem + p.L.nelem + p.R.nelem), "flops": reps * p.matvec_flops()}
    if kind == "batch":
        ps = [two_site("hubbard", D) for D in batch_dims(case)]
        return {"bytes": sum(4.0 * (2 * p.psi.nelem + p.L.nelem + p.R.nelem) for p in ps),
                "flops": sum(p.matvec_flops() for p in ps)}
    if kind == "env":
        p = two_site("xxz", case["D"])
        X = p.L if case["side"] == "left" else p.R
        return {"bytes": 8.0 * (2 * X.nelem + p.A.nelem), "flops": p.env_flops(case["side"])}
    # per site: the environment of H (about three dense channels' worth of blocks per charge) and
    # of the norm, forward and twice that backward
    flops = n = 0.0
    for legs in mps_legs(case["L"], case["D"]):
        n += legs.nelem
        by = {}
        for t, s in zip(legs.itoi.tolist(), legs.shapes.tolist()):
            by.setdefault(t[0], []).append(s)
        flops += 3.0 * 6.0 * sum(4.0 * s[0] * s[0] * s[2] for ss in by.values() for s in ss)
    return {"bytes": 16.0 * n, "flops": flops}


# About four times the largest relative error against `exact` (for the Lanczos vector: against the
# vector of `_exact_lanczos` up to its sign) seen over the drawn ranges and several seeds.
_REL = {
    "fp64": 2e-15,             # seen: 5.6e-16
    "mps": 2e-14,              # seen: 4.1e-15 (gradients, which cancel)
    "bf16x3": 3e-5,            # seen: 7.2e-6, the 16 significant bits of a split operand
    "3xtf32": 3e-5,            # seen: 7.8e-6, FP32 accumulation over K of a few thousand
    "batch_3xtf32": 4e-6,      # seen: 6e-7 (K of a few hundred)
    "lanczos_fp64": 3e-14,     # seen: 7e-15, the recurrence amplifies rounding
    "lanczos_bf16x3": 4e-4,    # seen: 9.4e-5
    "lanczos_3xtf32": 4e-5,    # seen: 8.2e-6
}


def tolerance(case):
    kind = case["kind"]
    if kind in ("permute", "blocks"):
        return "exact"
    if kind == "mps":
        return {"rel": _REL["mps"]}
    prec = case.get("precision", "fp64")
    key = f"{kind}_{prec}"
    return {"rel": _REL.get(key, _REL[prec])}


# ---------------------------------------------------------------- the same in float64, dense
def _dense_two_site(p, x, l, r):
    """A function psi -> H psi on dense tensors."""
    L, R, M = p.L.dense(l), p.R.dense(r), p.mpo_dense().to(l.device)
    Lt = L.transpose(1, 2).contiguous()  # [w, a', a]

    def apply(psi):  # [a, s1, s2, b]
        a, s1, s2, b = psi.shape
        w, xa = Lt.shape[0], Lt.shape[1]
        t = (Lt.reshape(w * xa, a) @ psi.reshape(a, -1)).view(w, xa, s1, s2, b)
        t = torch.einsum("wxstb,wvsy->vxytb", t, M)
        t = torch.einsum("vxytb,vutz->xyzub", t, M)
        return (t.reshape(xa * s1 * s2, -1) @ R.reshape(-1, R.shape[2])).view(xa, s1, s2, -1)

    return apply


def _exact_lanczos(apply, x, iters):
    """Plain three-term recurrence; the lowest Ritz pair, the vector as the combination of the
    Krylov vectors (its sign is fixed by a non-negative first coefficient)."""
    q = [x / torch.linalg.vector_norm(x)]
    al, be = [], []
    for i in range(iters):
        w = apply(q[-1])
        al.append(float((w * q[-1]).sum()))
        w = w - al[-1] * q[-1] - (be[-1] * q[-2] if i else 0.0)
        be.append(float(torch.linalg.vector_norm(w)))
        q.append(w / be[-1])
    T = np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1)
    ev, z = np.linalg.eigh(T)
    return float(ev[0]), sum(float(c) * v for c, v in zip(z[:, 0], q))


def exact(case, seed):
    kind = case["kind"]
    if kind == "permute":
        return _permute_input(case, seed).permute(*_ints(case["mapper"])).contiguous()
    if kind == "blocks":
        p, m = two_site(case["model"], case["D"]), _ints(case["mapper"])
        x = torch.from_numpy(p.vector(p.psi, np.random.default_rng(seed))).to(_device())
        return p.psi.permuted(m).flat(p.psi.dense(x).permute(*m))
    if kind == "dense_site":
        L, W, R, A = _dense_site_input(case, seed)
        t = torch.einsum("awx,asb->wxsb", L, A)
        t = torch.einsum("wxsb,wvsy->xyvb", t, W)
        return torch.einsum("xyvb,bvz->xyz", t, R)
    if kind == "heff":
        p = two_site("xxz", case["D"])
        x, l, r = _two_site_input(case, seed)
        return p.psi.flat(_dense_two_site(p, x, l, r)(p.psi.dense(x)))
    if kind == "lanczos":
        p = two_site("xxz", case["D"])
        x, l, r = _two_site_input(case, seed)
        E, v = _exact_lanczos(_dense_two_site(p, x, l, r), p.psi.dense(x), case["iters"])
        return {"energy": E, "vector": None}
    if kind == "batch":
        parts = []
        for D, data in zip(batch_dims(case), _batch_input(case, seed)):
            p = two_site("hubbard", D)
            x, l, r = (torch.from_numpy(d).to(_device()).double() for d in data)
            y = p.psi.flat(_dense_two_site(p, x, l, r)(p.psi.dense(x)))
            parts += [y, y.new_zeros(-len(y) % BATCH_ALIGN)]
        return torch.cat(parts)
    if kind == "env":
        p = two_site("xxz", case["D"])
        X, A = _env_input(case, seed)
        M, A = p.mpo_dense().to(X.device), p.A.dense(A)
        if case["side"] == "left":
            t = torch.einsum("wax,asb->wxsb", p.L.dense(X), A)
            t = torch.einsum("wxsb,wvst->vbxt", t, M)
            return p.L.flat(torch.einsum("vbxt,xty->vby", t, A))
        t = torch.einsum("asb,vby->asvy", A, p.R.dense(X))
        t = torch.einsum("asvy,wvst->waty", t, M)
        return p.R.flat(torch.einsum("waty,xty->wax", t, A))
    legs, flats = mps_legs(case["L"], case["D"]), _mps_input(case, seed)
    sites = [s.dense(x).requires_grad_(True) for s, x in zip(legs, flats)]
    M = two_site("xxz", 32).mpo_dense().to(flats[0].device)
    H, N = M.new_zeros(5, 1, 1), M.new_ones(1, 1)
    H[0, 0, 0] = 1.0
    for A in sites:
        t = torch.einsum("wax,asb->wxsb", H, A)
        t = torch.einsum("wxsb,wvst->vbxt", t, M)
        H = torch.einsum("vbxt,xty->vby", t, A)
        N = torch.einsum("axb,axc->bc", torch.einsum("ap,asb->psb", N, A), A)
    E = H[4, 0, 0] / N[0, 0]
    grads = torch.autograd.grad(E, sites)
    return {"energy": E.detach(), "gradient": [s.flat(g) for s, g in zip(legs, grads)]}
