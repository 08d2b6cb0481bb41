"""Performance cases: what a user of the engine has it do, through its public entry points.

The entry points are the Python mirror of the Julia interface (``kmhodlr``) and the C ABI of
``include/kmhodlr.h`` called on a handle that the program keeps, as a Julia program does.  Shapes
come from ``bench.py`` and the tests: points uniform on [0, 1]^2 in k-d order (iid normal for the
README's ACA example), Matern-3/2 or rational-quadratic kernels, Nystrom rank up to 80, leaves of
about 130 to 510 points, 1 to 32 right-hand sides, 8 to 72 probes, in the FP64 form (the default)
and in the mixed form.

``exact`` evaluates the same quantities with plain torch in 64 bits.  A Nystrom HODLR matrix with one
landmark set P is  K_H = Phi S^-1 Phi' + D,  Phi = K(X, P), S = K(P, P), D the diagonal leaves of
K - Phi S^-1 Phi'; D vanishes on the landmarks, so eliminating them first leaves a block-diagonal
matrix, which gives products, solves and the determinant.  The probes of the stochastic gradient
go through the symmetric factor W, built level by level.  ACA blocks approximate the dense matrix,
whose Cholesky factor is used.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kernelmatrices.jl_gb300"))

import kmhodlr as K  # noqa: E402
from kmhodlr import _lib as L  # noqa: E402
from kmhodlr.data import normal_points, uniform_points  # noqa: E402


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # one likelihood evaluation of an optimiser on a small data set: the smallest call, host included
        dict(name="objective_small", kind="objective", n=1000, rank=32, lv=8, kernel="matern32", range=0.1,
             nugget=1e-3, probes=24),
        # the same on an ordinary data set of odd size with the README's kernel
        dict(name="objective_ragged", kind="objective", n=10007, rank=72, lv=8, kernel="ratquad", range=0.2,
             nugget=1e-2, probes=72),
        # the headline step on resident data: assemble, product, factorise, 16 solves, logdet
        dict(name="step_mixed", kind="step", n=65536, rank=72, lv=8, kernel="matern32", range=0.1, nugget=1e-3,
             rhs=16, precision="mixed"),
        # the same in the plain FP64 form
        dict(name="step_fp64", kind="step", n=65536, rank=72, lv=8, kernel="matern32", range=0.1, nugget=1e-3,
             rhs=16, precision="fp64"),
        # a large likelihood with its gradient on a kept handle, the heavy request of a server
        dict(name="likelihood_large_mixed", kind="likelihood", n=250007, rank=72, lv=8, kernel="matern32", range=0.1,
             nugget=1e-3, probes=72, precision="mixed"),
        # an ordinary one in FP64
        dict(name="likelihood_fp64", kind="likelihood", n=30011, rank=72, lv=8, kernel="matern32", range=0.05,
             nugget=1e-3, probes=32, precision="fp64"),
        # kriging against a resident factor: one right-hand side, and a block of them
        dict(name="solve_one_mixed", kind="solve", n=131072, rank=72, lv=8, kernel="matern32", range=0.1,
             nugget=1e-3, rhs=1, precision="mixed"),
        dict(name="solve_block_fp64", kind="solve", n=40009, rank=64, lv=8, kernel="matern32", range=0.1,
             nugget=1e-3, rhs=32, precision="fp64"),
        # many independent data sets at once
        dict(name="batch_mixed", kind="batch", problems=24, lo=1024, hi=16384, rank=72, lv=8, kernel="matern32",
             nugget=1e-3, probes=72, precision="mixed"),
        # the README example: ACA to 1e-12, unsorted normal points, the diagonal raised by one
        dict(name="aca_readme", kind="aca", n=1024, lv=8, kernel="ratquad", points="normal", range=1.0, nugget=1.0,
             tol=1e-12, rhs=1),
        # ACA at an ordinary size: ranks of a few hundred at the top
        dict(name="aca_16k", kind="aca", n=16384, lv=8, kernel="matern32", points="uniform", range=0.05, nugget=1e-2,
             tol=1e-8, rhs=8),
        # gradient and Fisher information for scoring steps, on a resident factor
        dict(name="fisher_fp64", kind="fisher", n=8209, rank=48, lv=8, kernel="matern32", range=0.1, nugget=1e-3,
             probes=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["objective", "step", "step", "likelihood", "likelihood", "solve", "batch", "aca", "fisher"])
    case = dict(kind=kind, lv=8, kernel="matern32", nugget=rng.choice([1e-3, 1e-2]))
    if kind == "batch":
        case.update(problems=rng.randint(4, 24), lo=1024, hi=_log_int(rng, 2048, 16384), rank=rng.randint(24, 80),
                    probes=rng.randint(8, 72), precision=rng.choice(["fp64", "mixed"]))
        return case
    case["range"] = round(rng.uniform(0.04, 0.2), 3)
    if kind == "aca":
        if rng.random() < 0.5:
            case.update(n=_log_int(rng, 1024, 4096), kernel="ratquad", points="normal", range=1.0, nugget=1.0, tol=1e-12,
                        rhs=rng.randint(1, 8))
        else:
            case.update(n=_log_int(rng, 2048, 16384), points="uniform", nugget=1e-2, tol=1e-8, rhs=rng.randint(1, 8))
        return case
    case["rank"] = rng.randint(24, 80)
    if kind == "objective":
        case.update(n=_log_int(rng, 1000, 16384), kernel=rng.choice(["matern32", "ratquad"]), nugget=1e-2,
                    probes=rng.randint(8, 72))
    elif kind == "step":
        case.update(n=_log_int(rng, 2000, 65536), rhs=rng.randint(1, 16), precision=rng.choice(["fp64", "mixed"]))
    elif kind == "likelihood":
        case.update(precision=rng.choice(["fp64", "mixed"]), probes=rng.randint(8, 72))
        case["n"] = _log_int(rng, 4096, 250000 if case["precision"] == "mixed" else 65536)
    elif kind == "solve":
        case.update(n=_log_int(rng, 4096, 131072), rhs=rng.randint(1, 32), precision=rng.choice(["fp64", "mixed"]))
    else:
        case.update(n=_log_int(rng, 2048, 16384), probes=rng.randint(8, 32))
    return case


# ---- inputs and one pass -----------------------------------------------------------------------

KERNELS = {"matern32": K.Matern32(), "ratquad": K.RatQuad()}


def _params(case):
    return np.array([1.0, case.get("range", 0.1), case["nugget"]])


def _points(case, seed):
    n = case["n"]
    return normal_points(n, seed) if case.get("points") == "normal" else uniform_points(n, seed)


def _probes(n, count, seed):
    return np.asfortranarray(np.random.default_rng(seed).choice(np.array([-1.0, 1.0]), size=(n, count)))


def _observations(pts, seed):
    """A rough random field at the points plus noise: 256 random waves of heavy-tailed frequencies (a
    Matern-like spectrum of range 0.15) and N(0, 0.06^2)."""
    rng = np.random.default_rng(seed)
    w = rng.standard_normal((2, 256)) * np.sqrt(3.0 / rng.chisquare(3.0, 256)) / 0.15
    f = np.cos(pts @ w + rng.uniform(0, 2 * np.pi, 256)) @ rng.standard_normal(256)
    return f * np.sqrt(2.0 / 256) + 0.06 * rng.standard_normal(len(pts))


def _problems(case, seed):
    """(points, observations, parameters) of a batch: sizes spread over [lo, hi] on a log scale."""
    rng = np.random.default_rng(seed)
    m = case["problems"]
    out = []
    for b in range(m):
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((b + 0.5) / m)))
        rho = float(np.exp(rng.uniform(np.log(0.04), np.log(0.2))))
        pts = uniform_points(n, seed + 1 + b)
        out.append((pts, _observations(pts, seed + b), (1.0, rho, case["nugget"])))
    return out


def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double)) if isinstance(a, np.ndarray) else C.c_void_p(a.data_ptr())


class _Handle:
    """A C ABI handle that a program keeps between calls."""

    def __init__(self, case):
        cfg = L.KmConfig(device=0, precision=L.KM_PREC_MIXED if case["precision"] == "mixed" else L.KM_PREC_FP64,
                         hbm_budget_fraction=0.8, refine_max_iter=0, refine_tol=0.0)
        self.lib = L.load()
        self.h = C.c_void_p()
        if self.lib.km_create(C.byref(cfg), C.byref(self.h)) != L.KM_OK:
            raise RuntimeError("km_create failed")
        self.case, self.params = case, _params(case)

    def __call__(self, name, *args):
        if getattr(self.lib, name)(self.h, *args) != L.KM_OK:
            raise RuntimeError(self.lib.km_last_error(self.h).decode())

    def assemble(self, pts):
        c = self.case
        self("km_assemble" if isinstance(pts, np.ndarray) else "km_assemble_dev", _ptr(pts), c["n"],
             KERNELS[c["kernel"]].kid, _ptr(self.params), 3, L.KM_METHOD_NYSTROM, 0.0, c["rank"], L.KM_LEVEL_LOG, c["lv"])

    def __del__(self):
        if self.h:
            self.lib.km_destroy(self.h)
            self.h = None


def _step_inputs(case, seed):
    """Points, a vector and right-hand sides (row c is column c) on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    pts = torch.from_numpy(_points(case, seed)).cuda()
    x = torch.randn(case["n"], dtype=torch.float64, device="cuda", generator=g)
    b = torch.randn(case["rhs"], case["n"], dtype=torch.float64, device="cuda", generator=g)
    return pts, x, b


def _aca_rhs(case, seed):
    return np.asfortranarray(np.random.default_rng(seed).standard_normal((case["n"], case["rhs"])))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed)
    if kind == "batch":
        s["problems"] = [K.Problem(*p) for p in _problems(case, seed)]
        s["engine"] = K.BatchEngine(precision=L.KM_PREC_MIXED if case["precision"] == "mixed" else L.KM_PREC_FP64)
        return s
    if kind in ("step", "solve"):
        s["pts"], s["x"], s["b"] = _step_inputs(case, seed)
        s["y"], s["sol"] = torch.empty_like(s["x"]), torch.empty_like(s["b"])
        s["handle"] = _Handle(case)
        torch.cuda.synchronize()  # the handle has a stream of its own
        if kind == "solve":
            s["handle"].assemble(s["pts"])
            s["handle"]("km_factorize")
        return s
    s["pts"] = _points(case, seed)
    if kind == "aca":
        s["rhs"] = _aca_rhs(case, seed)
        return s
    s["data"] = _observations(s["pts"], seed)
    if kind == "likelihood":
        s["handle"] = _Handle(case)
    elif kind == "objective":
        s["probes"] = _probes(case["n"], case["probes"], seed + 1)
    else:
        s["hk"] = K.KernelHODLR(K.KernelMatrix(s["pts"], s["pts"], _params(case), KERNELS[case["kernel"]]), 0.0,
                                case["rank"], K.LogLevel(case["lv"]), nystrom=True)
        K.symmetricfactorize(s["hk"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "objective":
        grad = np.zeros(3)
        nll = K.nll_objective(_params(case), grad, s["pts"], s["data"], KERNELS[case["kernel"]], case["rank"],
                              K.LogLevel(case["lv"]), s["probes"])
        return {"nll": nll, "grad": grad}
    if kind == "step":
        h, ld = s["handle"], C.c_double()
        h.assemble(s["pts"])
        h("km_matvec_dev", _ptr(s["x"]), _ptr(s["y"]), 1)
        h("km_factorize_solve_dev", _ptr(s["b"]), _ptr(s["sol"]), case["rhs"])
        h("km_logdet", C.byref(ld))
        return {"product": s["y"], "solution": s["sol"], "logdet": ld.value}
    if kind == "likelihood":
        h, nll, grad = s["handle"], C.c_double(), np.zeros(3)
        h.assemble(s["pts"])
        h("km_factorize")
        h("km_nll_grad_seeded", _ptr(s["data"]), case["probes"], s["seed"], C.byref(nll), _ptr(grad))
        return {"nll": nll.value, "grad": grad}
    if kind == "solve":
        s["handle"]("km_solve_dev", _ptr(s["b"]), _ptr(s["sol"]), case["rhs"])
        return {"solution": s["sol"]}
    if kind == "batch":
        nll, grad, _ = s["engine"].nll_grad(s["problems"], KERNELS[case["kernel"]], case["rank"], K.LogLevel(case["lv"]),
                                            nprobe=case["probes"], seed=s["seed"])
        return {"nll": nll, "grad": grad}
    if kind == "aca":
        hk = K.KernelHODLR(K.KernelMatrix(s["pts"], s["pts"], _params(case), KERNELS[case["kernel"]]), case["tol"], 0,
                           K.LogLevel(case["lv"]))
        y = hk @ s["rhs"]
        K.symmetricfactorize(hk)
        return {"product": y, "solution": hk.ldiv(s["rhs"]), "logdet": hk.logdet()}
    nll, grad, fisher = K.grad_and_fisher(s["hk"], s["data"], nprobe=case["probes"], seed=s["seed"])
    return {"nll": nll, "grad": grad, "fisher": fisher}


# ---- the work of one pass ----------------------------------------------------------------------

def _levels(n, lv):
    return max(0, n.bit_length() - 1 - lv)


def _nystrom_work(case, n, rhs, probes, factor=True, scorings=0):
    """Leaf Cholesky, leaf panels and their bases, r x r node work, solves and derivative forms."""
    r, m = case["rank"], n / 2 ** _levels(n, case["lv"])
    nodes = 2 ** _levels(n, case["lv"]) - 1
    cols = rhs + probes
    f = (n * m * m / 3 + n * m * r + 2 * n * r * r + 7 * nodes * r ** 3 + 20 * n * (m / 2 + r)) if factor else 0
    f += rhs * 2 * (n * m + 4 * n * r + 8 * nodes * r * r)
    f += probes * (n * m + 4 * n * r + 8 * nodes * r * r + n * m + 6 * n * r)
    f += scorings * probes * (3 * n * m + 6 * n * r)
    return {"bytes": 8.0 * n * (2 + 2 * max(1, cols if rhs else 1)), "flops": float(f)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = []
        for b in range(case["problems"]):
            n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((b + 0.5) / case["problems"])))
            ws.append(_nystrom_work(case, n, 1, case["probes"]))
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    n = case["n"]
    if kind == "solve":
        # the factor is read once whatever the number of right-hand sides
        w = _nystrom_work(case, n, case["rhs"], 0, factor=False)
        m = n / 2 ** _levels(n, case["lv"])
        return {"bytes": w["bytes"] + 8.0 * n * (m / 2 + case["rank"]), "flops": w["flops"]}
    if kind == "aca":
        # ranks are known after the pass only: leaf Cholesky and a rank of 32 on every level
        m, lev, q = n / 2 ** _levels(n, case["lv"]), _levels(n, case["lv"]), 32
        f = n * m * m / 3 + n * lev * q * (m + 6 * q * lev) + case["rhs"] * 2 * n * (m + 4 * q * lev)
        return {"bytes": 8.0 * n * (2 + 3 * case["rhs"]), "flops": float(f)}
    if kind == "fisher":
        return _nystrom_work(case, n, 1, case["probes"], factor=False, scorings=3)
    if kind == "step":
        return _nystrom_work(case, n, case["rhs"] + 1, 0)
    return _nystrom_work(case, n, 1, case["probes"])


# ---- the same in 64 bits -----------------------------------------------------------------------

def _kernel(kernel, p, x, y, deriv=None):
    """k(x, y), or its derivative in parameter `deriv`, for (..., a, 2) against (..., b, 2) points."""
    d = x.unsqueeze(-2) - y.unsqueeze(-3)
    r = (d * d).sum(-1).sqrt()
    same = (d == 0).all(-1).to(r.dtype)
    if deriv == 2:
        return same
    if kernel == "ratquad":
        u = 1 + (r / p[1]) ** 2
        if deriv == 0:
            return 2 * p[0] / u ** 2
        if deriv == 1:
            return 4 * p[0] ** 2 * r ** 2 / (p[1] ** 3 * u ** 3)
        return p[0] ** 2 / u ** 2 + p[2] * same
    z = math.sqrt(3.0) * r / p[1]
    e = torch.exp(-z)
    if deriv == 0:
        return (1 + z) * e
    if deriv == 1:
        return p[0] * z * z * e / p[1]
    return p[0] * (1 + z) * e + p[2] * same


class _Exact:
    """A Nystrom HODLR matrix: leaves padded to one size (zero rows of Phi, identity rows of K)."""

    def __init__(self, pts, p, kernel, rank, lv):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.kernel, self.r = [float(v) for v in p], kernel, rank
        X = torch.as_tensor(pts, dtype=torch.float64, device=dev)
        n = self.n = X.shape[0]
        lev = self.lev = _levels(n, lv)
        nl = 2 ** lev
        m0, rem = n // nl, n % nl
        m = self.m = m0 + (rem > 0)
        start = torch.arange(nl, device=dev) * m0 + torch.arange(nl, device=dev).clamp(max=rem)
        size = m0 + (torch.arange(nl, device=dev) < rem)
        at = start[:, None] + torch.arange(m, device=dev)
        self.live = torch.arange(m, device=dev) < size[:, None]
        self.at = torch.where(self.live, at, torch.zeros_like(at))
        t = torch.arange(rank, dtype=torch.float64) / (rank - 1)
        self.lnd = ((1 - t) + t * n).round().long().to(dev) - 1
        self.P, self.X = X[self.lnd], X[self.at]
        self.S = _kernel(kernel, self.p, self.P, self.P)
        self.Sc = torch.linalg.cholesky(self.S)
        self.Phi = self._phi()
        self.both = self.live[:, :, None] & self.live[:, None, :]
        self.Kl = self._leaves()

    def _leaves(self, deriv=None):
        k = _kernel(self.kernel, self.p, self.X, self.X, deriv)
        return torch.where(self.both, k, torch.eye(self.m, dtype=k.dtype, device=k.device) if deriv is None else 0 * k)

    def _phi(self, deriv=None):
        return torch.where(self.live[:, :, None], _kernel(self.kernel, self.p, self.X, self.P, deriv), 0.0)

    def pad(self, x):  # (n, k) -> (leaves, m, k)
        return torch.where(self.live[:, :, None], x[self.at], 0.0)

    def unpad(self, x):
        out = torch.empty(self.n, x.shape[-1], dtype=x.dtype, device=x.device)
        out[self.at[self.live]] = x[self.live]
        return out

    def eliminate(self):
        """D with unit rows at the landmarks, its Cholesky factor, and the landmarks' places."""
        V = torch.linalg.solve_triangular(self.Sc, self.Phi.mT.reshape(self.Phi.shape[0], self.r, self.m), upper=False)
        self.D = self.Kl - torch.where(self.both, V.mT @ V, 0.0)
        mark = torch.zeros(self.n, dtype=torch.bool, device=self.D.device)
        mark[self.lnd] = True
        self.free = self.live & ~mark[self.at]
        keep = self.free[:, :, None] & self.free[:, None, :]
        self.D = torch.where(keep, self.D, 0.0)
        self.Dc = torch.linalg.cholesky(torch.where(keep, self.D, torch.eye(self.m, dtype=self.D.dtype, device=self.D.device)))

    def mul(self, x):
        xl = self.pad(x)
        g = torch.cholesky_solve((self.Phi.mT @ xl).sum(0), self.Sc)
        return self.unpad(self.D @ xl + self.Phi @ g)

    def solve(self, b):
        bP = b[self.lnd]
        bl = torch.where(self.free[:, :, None], self.pad(b) - self.Phi @ torch.cholesky_solve(bP, self.Sc), 0.0)
        xl = torch.cholesky_solve(bl, self.Dc)
        x = self.unpad(xl)
        x[self.lnd] = torch.cholesky_solve(bP - (self.Phi.mT @ xl).sum(0), self.Sc)
        return x

    def logdet(self):
        return float(2 * self.Sc.diagonal().log().sum() + 2 * self.Dc.diagonal(dim1=-2, dim2=-1).log().sum())

    def factor(self):
        """Leaf factors and, per level, the children's orthonormal bases with Ct and L22."""
        self.Lc = torch.linalg.cholesky(self.Kl)
        A = torch.linalg.solve_triangular(self.Lc, self.Phi, upper=False)
        self.nodes = []
        eye = torch.eye(self.r, dtype=A.dtype, device=A.device)
        for _ in range(self.lev):
            Q, R = torch.linalg.qr(A)
            Q1, Q2, R1, R2 = Q[0::2], Q[1::2], R[0::2], R[1::2]
            Ct = R1 @ torch.cholesky_solve(R2.mT, self.Sc.expand_as(R2))
            L22 = torch.linalg.cholesky(eye - Ct.mT @ Ct)
            self.nodes.append((Q1, Q2, Ct, L22))
            A = torch.cat([Q1 @ R1, Q2 @ torch.linalg.solve_triangular(L22, R2 - Ct.mT @ R1, upper=False)], 1)

    def half(self, v, transpose):
        """W^-1 v, or W'^-1 v."""
        x = self.pad(v)
        nl, m, k = x.shape
        if not transpose:
            x = torch.linalg.solve_triangular(self.Lc, x, upper=False)
        for Q1, Q2, Ct, L22 in (reversed(self.nodes) if transpose else self.nodes):
            x = x.reshape(Q1.shape[0], 2, -1, k)
            z2 = Q2.mT @ x[:, 1]
            if transpose:
                w = torch.linalg.solve_triangular(L22.mT, z2, upper=True)
                x = torch.stack([x[:, 0] - Q1 @ (Ct @ w), x[:, 1] - Q2 @ (z2 - w)], 1)
            else:
                w = torch.linalg.solve_triangular(L22, z2 - Ct.mT @ (Q1.mT @ x[:, 0]), upper=False)
                x = torch.stack([x[:, 0], x[:, 1] - Q2 @ (z2 - w)], 1)
        x = x.reshape(nl, m, k)
        if transpose:
            x = torch.linalg.solve_triangular(self.Lc.mT, x, upper=True)
        return self.unpad(x)

    def derivatives(self, x):
        """dK_j x for the three parameters: exact leaves, the derivative of Phi S^-1 Phi' elsewhere."""
        xl = self.pad(x)
        out = []
        for j in range(3):
            dPhi, Sj = self._phi(j), _kernel(self.kernel, self.p, self.P, self.P, j)
            a, b = self.Phi.mT @ xl, dPhi.mT @ xl
            a, b = a.sum(0) - a, b.sum(0) - b  # every leaf against all others
            u = torch.cholesky_solve(a, self.Sc.expand(a.shape[0], -1, -1))
            w = torch.cholesky_solve(b - Sj @ u, self.Sc.expand(a.shape[0], -1, -1))
            out.append(self.unpad(self._leaves(j) @ xl + dPhi @ u + self.Phi @ w))
        return out

    def likelihood(self, y, probes, fisher=False):
        self.eliminate()
        self.factor()
        y = torch.as_tensor(y, dtype=torch.float64, device=self.S.device)[:, None]
        probes = torch.as_tensor(np.ascontiguousarray(probes), dtype=torch.float64, device=self.S.device)
        alpha = self.solve(y)
        nll = 0.5 * (self.logdet() + float((y * alpha).sum()))
        T = self.half(probes, True)
        dT, da = self.derivatives(T), self.derivatives(alpha)
        grad = [0.5 * float((T * dT[j]).sum() / T.shape[1] - (alpha * da[j]).sum()) for j in range(3)]
        if not fisher:
            return nll, grad
        U = [self.half(d, False) for d in dT]
        return nll, grad, [[0.5 * float((U[j] * U[k]).sum()) / T.shape[1] for k in range(3)] for j in range(3)]


def _mix64(x):
    with np.errstate(over="ignore"):
        z = x + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _seeded_probes(n, count, seed):
    """+1 where the top bit of SplitMix64(SplitMix64(seed) + j n + i) is set, else -1."""
    with np.errstate(over="ignore"):
        e = _mix64(np.array([seed], dtype=np.uint64))[0] + np.arange(n * count, dtype=np.uint64)
    return np.where(_mix64(e) >> np.uint64(63) == 1, 1.0, -1.0).reshape(count, n).T


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        nll, grad = [], []
        for b, (pts, y, p) in enumerate(_problems(case, seed)):
            e = _Exact(pts, p, case["kernel"], case["rank"], case["lv"])
            v, g = e.likelihood(y, _seeded_probes(len(y), case["probes"], seed + b))
            nll.append(v)
            grad.append(g)
        return {"nll": np.array(nll), "grad": np.array(grad)}
    if kind == "aca":
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        b = torch.from_numpy(_aca_rhs(case, seed)).to(dev)
        X = torch.from_numpy(_points(case, seed)).to(dev)
        A = _kernel(case["kernel"], _params(case).tolist(), X, X)
        y, Lc = (A @ b).cpu().numpy(), torch.linalg.cholesky(A)
        return {"product": y, "solution": torch.cholesky_solve(b, Lc).cpu().numpy(),
                "logdet": float(2 * Lc.diagonal().log().sum())}
    if kind in ("step", "solve"):
        pts, x, b = _step_inputs(case, seed)
        e = _Exact(pts, _params(case), case["kernel"], case["rank"], case["lv"])
        e.eliminate()
        sol = e.solve(b.T).T.contiguous()
        if kind == "solve":
            return {"solution": sol}
        return {"product": e.mul(x[:, None])[:, 0], "solution": sol, "logdet": e.logdet()}
    pts, n = _points(case, seed), case["n"]
    y = _observations(pts, seed)
    e = _Exact(pts, _params(case), case["kernel"], case["rank"], case["lv"])
    if kind == "fisher":
        nll, grad, F = e.likelihood(y, _seeded_probes(n, case["probes"], seed), fisher=True)
        return {"nll": nll, "grad": np.array(grad), "fisher": np.array(F)}
    V = _probes(n, case["probes"], seed + 1) if kind == "objective" else _seeded_probes(n, case["probes"], seed)
    nll, grad = e.likelihood(y, V)
    return {"nll": nll, "grad": np.array(grad)}
