"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values. ``prepare`` makes what a program has in hand before the call
(data on the host, an open context at the state the call starts from), ``run`` makes ONE pass
through the public entry points (``gaspacho2_b200``) and returns its outputs, ``exact`` gives the
same outputs in float64 with plain torch, and ``work`` the bytes and operations that a pass cannot
do without. Sizes follow the configurations of ``gaspacho2_b200.synth`` (0: 2,000 cells x 500
genes; 1: 20,000 x 2,000; 2: 100,000 x 10,000 with 100 donors; 4: 300 donors and 256 inducing
points), with odd and ragged ones among them and fewer genes where a pass would take too long.

The data are synthetic counts at a state near the end of a fit: cells at unit-variance latent
coordinates, inducing points spread over them, length-scales between the generator's and the start's,
and counts drawn from the model's own rates.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from gaspacho2_b200 import _lib, de, encoder
from gaspacho2_b200.formats import Counts, Design, Params
from gaspacho2_b200.model import GPLVM

F64 = torch.float64
WT, IGA, IGB = 0.1, 100.0, 100.0  # Titsias weight and the inverse-gamma prior on Omega


def listed():
    return [
        # one objective + gradient evaluation (the unit of the headline metric) through host
        # parameters. Configuration 0: what a trial run or a test does, bound by launches
        dict(name="evaluate small", kind="evaluate", N=2000, J=500, M=32, Q=2, batch=2, num=1, donors=0,
             precision="fp64", graph=0),
        # configuration 1, ragged in cells and genes, evaluations replayed as graphs
        dict(name="evaluate medium", kind="evaluate", N=19997, J=1999, M=64, Q=5, batch=4, num=3, donors=0,
             precision="fp64", graph=1),
        # configuration 2's cells, design and model: the headline shape with fewer genes
        dict(name="evaluate large", kind="evaluate", N=100000, J=3000, M=128, Q=10, batch=4, num=3, donors=100,
             precision="fp64", graph=1),
        # the same in the tensor-core form that the user may choose
        dict(name="evaluate bf16x3", kind="evaluate", N=50000, J=2000, M=128, Q=10, batch=4, num=3, donors=100,
             precision="bf16x3", graph=1),
        # configuration 4's design: 300 donors, 256 inducing points (P = 564 model columns)
        dict(name="evaluate wide", kind="evaluate", N=30011, J=501, M=256, Q=10, batch=4, num=3, donors=300,
             precision="fp64", graph=0),
        # the start of a fit: kernel matrices, GLM coefficients and an IRLS sweep
        dict(name="irls", kind="irls", N=60000, J=2001, M=128, Q=10, batch=4, num=3, donors=100, sweep=30,
             fused_tail=1),
        # the start of a small fit phase by phase, as the drivers call them: GLM coefficients, IRLS
        # sweeps, the objective, its gradient, an L-BFGS step and the objective there
        dict(name="fit small", kind="fit", N=3001, J=301, M=32, Q=2, batch=2, num=1, donors=0, sweeps=20),
        # the differential-expression driver's model comparison on open contexts
        dict(name="model comparison", kind="de", N=20000, J=1001, M=64, Q=5, batch=4, num=3, donors=48, reduced=5,
             sweeps=2),
        # genotypes against a fitted model: shared columns and each gene's own cis variants
        dict(name="genotype statistics", kind="scores", N=30000, J=1000, M=128, Q=10, batch=4, num=3, donors=100,
             columns=20, variants=20),
        # new cells placed at a fitted model
        dict(name="placement", kind="place", N=20003, J=2000, M=128, Q=10, batch=4, num=3, donors=0, steps=3),
        # the amortised encoder: an epoch of training and the prediction of held-out cells
        dict(name="encoder", kind="encoder", N=16384, J=2000, M=32, Q=10, batch=4, num=3, donors=0, hidden=256,
             rows=1024, held=50001),
        # the kernel matrices alone on device memory, as a host framework's plugin calls them
        dict(name="kernel matrices", kind="kernels", N=100000, M=128, Q=10),
    ]


# ---- drawn cases ---------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "evaluate", "irls", "irls", "fit", "de", "scores",
                       "place", "encoder", "kernels"])
    Q = rng.choice([2, 5, 10])
    M = {2: rng.randint(8, 32), 5: rng.randint(16, 64), 10: rng.choice([rng.randint(32, 128), rng.randint(128, 256)])}[Q]
    N = _log_int(rng, 1000, 100000)
    if kind == "kernels":
        return dict(kind=kind, N=N, M=M, Q=Q)
    c = dict(kind=kind, N=N, J=_log_int(rng, 100, 3000), M=M, Q=Q, batch=rng.randint(2, 6), num=rng.randint(1, 4),
             donors=rng.choice([0, rng.randint(8, 100), rng.randint(100, 300)]) if N >= 8000 else 0)
    if kind == "evaluate":
        c.update(precision="bf16x3" if M <= 128 and rng.random() < 0.2 else "fp64", graph=rng.randint(0, 1))
    elif kind == "irls":
        c.update(sweep=rng.randint(0, 60), fused_tail=rng.randint(0, 1))
    elif kind == "fit":
        c.update(N=min(N, 5000), J=min(c["J"], 500), donors=0, sweeps=rng.randint(5, 20))
    elif kind == "de":
        c.update(reduced=rng.randint(4, 8), sweeps=rng.randint(1, 3))
    elif kind == "scores":
        c.update(donors=rng.randint(20, 100), N=max(N, 4000), M=min(M, 128), columns=rng.randint(1, 40), variants=rng.randint(1, 30))
    elif kind == "place":
        c.update(donors=0, steps=rng.randint(1, 4))
    elif kind == "encoder":
        c.update(N=max(N, 2048), donors=0, hidden=rng.choice([128, 256, 384]), rows=rng.choice([256, 512, 1024]),
                 held=_log_int(rng, 1000, 50000), M=8)
    return c


def draw(rng):
    most = work(listed()[2])
    while True:
        c = _draw_once(rng)
        w = work(c)
        if w["flops"] <= 0.5 * most["flops"] and w["bytes"] <= 0.7 * most["bytes"] and c["N"] * c.get("J", 0) <= 2e8:
            return c


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    c = dict(case)
    N, M, Q, kind = c["N"], c["M"], c["Q"], c["kind"]
    if kind == "kernels":  # Knm and Kmm^-1 k_n of every cell
        return {"bytes": 8.0 * (N * Q + 2 * N * M + N), "flops": 2.0 * N * M * M + 3.0 * N * M * Q}
    J = c["J"]
    n_d = 1 + c["num"] + M  # dense model columns
    P = n_d + c["batch"] + c["donors"]
    nz = 0.2 * N * J
    gram = 1.0 * N * J * n_d * (n_d + 1)  # the symmetric half, multiply and add
    pred = 2.0 * N * J * n_d
    chol = J * P ** 3 / 3.0
    data = 8.0 * N * J + 12.0 * nz + 8.0 * N * n_d
    if kind == "evaluate":  # Gram, Z^T u, predictions, the group sums both ways, C1; Cholesky and inverse
        return {"bytes": 16.0 * N * J + 16.0 * N * Q + 16.0 * J * P, "flops": 2 * gram + 6 * pred + 3 * chol}
    if kind in ("irls", "de"):
        models = 1 if kind == "irls" else c["sweeps"]
        b, f = data + 16.0 * J * P, gram + 4 * pred + chol
        if kind == "de":  # the per-dimension models have a few GP columns
            r = 1 + c["num"] + c["reduced"]
            f += (Q + 1) * (1.0 * N * J * r * (r + 1) + 8.0 * N * J * r)
            b *= Q + 2
        return {"bytes": b * models, "flops": f * models}
    if kind == "fit":
        k = c["sweeps"] + 2
        return {"bytes": data * k, "flops": k * (gram + 4 * pred + chol)}
    if kind == "scores":
        L, V = c["columns"], c["variants"]
        return {"bytes": data + 8.0 * N * L + 8.0 * J * (L + 2 * V),
                "flops": 2.0 * N * J * n_d * L + 2 * pred + 2.0 * J * P * P * (L + V)}
    if kind == "place":
        return {"bytes": (data + 8.0 * N * Q) * (2 * c["steps"] + 2), "flops": (4 * c["steps"] + 4) * pred}
    n_in, H = c["J"], c["hidden"]  # encoder
    mlp = 2.0 * (n_in * H + H * H + H * 2 * Q)
    return {"bytes": 2.0 * (3 * N + c["held"]) * n_in, "flops": mlp * (3 * N + c["held"])}


# ---- data --------------------------------------------------------------------------------------------
def _np(t):
    return t.cpu().numpy()


def _kernel(A, B, rho):
    """Periodic in dimension 0, ARD in the others."""
    s = torch.sin((A[:, None, 0] - B[None, :, 0]) / 2.0) ** 2 / rho[0]
    for q in range(1, A.shape[1]):
        s = s + (A[:, None, q] - B[None, :, q]) ** 2 / 2.0 / rho[q]
    return torch.exp(-s)


def _spread(X, M, rho):
    """M inducing points among the cells X, each the farthest from those before it in the kernel's metric."""
    near = torch.zeros(X.shape[0], dtype=F64, device="cuda")
    at = torch.zeros((), dtype=torch.int64, device="cuda")
    picked = []
    for _ in range(M):
        picked.append(at)
        near = torch.maximum(near, _kernel(X, X[at][None, :], rho)[:, 0])
        at = near.argmin()
    return X[torch.stack(picked)].clone()


def _rho(Q):
    """Length-scales between the generator's (1) and the start's (5, 10, ..): shorter in few dimensions."""
    f = {2: 0.1, 5: 0.3}.get(Q, 0.5)
    return np.array([5.0 * f] + [10.0 * f] * (Q - 1))


class _World:
    """The model at its parameters and the counts drawn from it, on the GPU, from the seed alone."""

    def __init__(self, c, seed, N=None, counts=True):
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
        self.g = g
        N = N or c["N"]
        J, M, Q = c["J"], c["M"], c["Q"]
        self.N, self.J, self.M, self.Q = N, J, M, Q
        rn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=F64)  # noqa: E731
        self.rn = rn
        self.X = rn(N, Q)
        self.rho = torch.tensor(_rho(Q), device="cuda")
        self.T = _spread(self.X[:2048], M, self.rho)
        self.s = torch.exp(0.3 * rn(N))
        self.batch = torch.randint(0, c["batch"], (N,), generator=g, device="cuda")
        self.numeric = rn(N, c["num"])
        nd = c["donors"]
        self.donor = torch.randint(0, nd, (N,), generator=g, device="cuda") if nd else None
        p = 2 + 1 + c["num"] + (1 if nd else 0)
        d = np.full(p, 0.05)
        d[0], d[-1] = 1.5, 0.3
        self.delta = torch.tensor(d, device="cuda")
        self.Omega = torch.exp(0.1 * rn(N))
        cols = [torch.ones(N, 1, dtype=F64, device="cuda"), torch.nn.functional.one_hot(self.batch, c["batch"]).to(F64),
                self.numeric]
        self.widths = [1, c["batch"]] + [1] * c["num"]
        if nd:
            cols.append(torch.nn.functional.one_hot(self.donor, nd).to(F64))
            self.widths.append(nd)
        self.C = torch.cat(cols, 1)  # covariate columns
        K = _kernel(self.X, self.T, self.rho)
        nc = self.C.shape[1]
        beta = torch.cat([(rn(1, J) * 1.2 - 2.0), 0.2 * rn(c["batch"] + c["num"], J)]
                         + ([0.3 * rn(nd, J)] if nd else [])
                         + [rn(M, J) / torch.sqrt((K * K).sum(1).mean())], 0)
        self.beta, self.P = beta, nc + M  # P x J
        if not counts:
            return
        Z = torch.cat([self.C, K], 1).float()
        bf = beta.float()
        ci, cx, per = [], [], []
        step = max(1, 20_000_000 // N)
        for j in range(0, J, step):
            lam = torch.exp(bf[:, j:j + step].T @ Z.T) * self.s.float()[None, :]
            y = torch.poisson(lam, generator=g)
            at = y.nonzero()
            per.append(torch.bincount(at[:, 0], minlength=y.shape[0]))
            ci.append(at[:, 1].int())
            cx.append(y[at[:, 0], at[:, 1]].double())
        self.cell, self.count = torch.cat(ci), torch.cat(cx)
        self.ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cat(per).cumsum(0)])

    def counts(self):
        return Counts(self.N, self.J, _np(self.cell), _np(self.ptr).astype(np.int32), _np(self.count))

    def design(self):
        N, nd = self.N, self.donor is not None
        lev = [self.widths[1]] + [1] * self.numeric.shape[1] + ([self.widths[-1]] if nd else [])
        cols = [_np(self.batch).astype(np.int32)]
        cols += [_np(self.numeric[:, k:k + 1]) for k in range(self.numeric.shape[1])]
        if nd:
            cols.append(_np(self.donor).astype(np.int32))
        return Design(N, np.array(lev, np.int32), np.ones(len(lev), np.int32), cols)

    def params(self):
        return Params(_np(self.Omega), _np(self.delta), _np(self.X), _np(self.T), _np(self.rho), np.ones(self.J))

    def moved(self):
        """The parameters of a line-search trial near the state, [Omega | delta | X | T | rho]."""
        rn = self.rn
        m = [self.Omega * torch.exp(0.01 * rn(self.N)), self.delta * torch.exp(0.01 * rn(len(self.delta))),
             self.X + 0.01 * rn(self.N, self.Q), self.T + 0.01 * rn(self.M, self.Q),
             self.rho * torch.exp(0.01 * rn(self.Q))]
        return m

    def context(self, c, precision="fp64"):
        m = GPLVM(self.counts(), self.design(), _np(self.s), _np(self.X), self.M, self.Q, precision=precision)
        m.set_params(self.params())
        return m


def _flat(parts):
    return np.concatenate([_np(t.T.contiguous().ravel() if t.dim() == 2 else t) for t in parts])


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "kernels":
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
        N, M, Q = c["N"], c["M"], c["Q"]
        e = lambda *s: torch.empty(*s, dtype=F64, device="cuda")  # noqa: E731
        X = torch.randn(Q, N, generator=g, device="cuda", dtype=F64)  # column-major N x Q
        rho = torch.tensor(_rho(Q), device="cuda")
        T = _spread(X.T[:2048], M, rho).T.contiguous()
        return dict(kind=kind, N=N, M=M, Q=Q, X=X, T=T, rho=rho, Knm=e(M, N),
                    Kinv=e(M, N), tit=e(N), lib=_lib.load())
    if kind == "encoder":
        w, h = _World(c, seed), _World(c, seed + 1000003, N=c["held"])
        enc = encoder.Encoder(c["J"], c["Q"], hidden=c["hidden"], batch=c["rows"], seed=1)
        genes = np.arange(c["J"], dtype=np.int32)
        order = np.random.default_rng(seed).permutation(c["N"]).astype(np.int32)
        enc.set_cells(0, w.counts(), _np(w.s), genes, order)
        enc.set_targets(_np(w.X))
        enc.set_cells(1, h.counts(), _np(h.s), genes)
        return dict(kind=kind, enc=enc)
    w = _World(c, seed)
    if kind == "de":
        ctx = de.open_contexts(w.counts(), w.design(), _np(w.s), _np(w.X), c["Q"], c["reduced"], c["M"])
        return dict(kind=kind, case=c, y=Counts(w.N, w.J, None, None, None), ls=_np(w.s), prm=w.params(), ctx=ctx)
    m = w.context(c, c.get("precision", "fp64"))
    s = dict(kind=kind, case=c, m=m)
    if kind == "irls":
        m.set_option("fused_tail", c["fused_tail"])
    elif kind == "fit":
        s["prm"] = w.params()
    elif kind == "place":
        m.set_beta(_np(w.beta))
        s["X0"] = _np(w.X + 0.3 * w.rn(w.N, w.Q))
    else:  # evaluate, scores: W and nu as an IRLS sweep leaves them
        m.set_beta(_np(w.beta))
        m.kernel_mats()
        m.expand_delta()
        m.irls_sweep(0, 0)
        if kind == "evaluate":
            m.set_option("graph", c["graph"])
            s["params"], s["grad"] = _flat(w.moved()), np.zeros(m.n_params())
        else:
            s["G"] = _np(torch.randint(0, 3, (c["columns"], w.N), generator=w.g, device="cuda").double()).T
            s["dos"] = _np(torch.randint(0, 3, (c["donors"], w.J, c["variants"]), generator=w.g, device="cuda").to(torch.int8))
    return s


# ---- one pass --------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "evaluate":
        obj, grad = s["m"].evaluate(s["params"], s["grad"])
        return {"objective": np.float64(obj), "gradient": grad}
    if kind == "irls":
        m = s["m"]
        m.kernel_mats()
        m.glm_init()
        lk = m.irls_sweep(0, s["case"]["sweep"])
        return {"likelihood": np.float64(lk), "beta": m.get("Beta"), "phi": m.get("phi")}
    if kind == "fit":
        m = s["m"]
        m.set_params(s["prm"])
        m.kernel_mats()
        m.glm_init()
        n = m.irls(0, s["case"]["sweeps"])
        first = m.objective_after_irls()
        grad = m.gradient()
        m.lbfgs_update(0, 0)
        return {"sweeps": n, "objective": np.float64(first), "gradient": grad, "step": np.float64(m.objective(0, 1)), "X": m.get("X"),
                "Omega": m.get("Omega"), "beta": m.get("Beta")}
    if kind == "de":
        c = s["case"]
        r = de.de_bfs(s["y"], None, s["ls"], s["prm"], c["Q"], c["reduced"], c["M"], jtr_max=c["sweeps"],
                      contexts=s["ctx"])
        return {"BFs": r["BFs"], "phi": r["phi"]}
    if kind == "scores":
        m, c = s["m"], s["case"]
        S = m.score_stats(s["G"])
        cis, lr = m.cis_stats(s["dos"], c["num"] + 1)
        return {"S": S, "cis": cis, "LR": lr}
    if kind == "place":
        o, g = encoder.cell_objective(s["m"], s["X0"], grad=True)
        X, obj, st = encoder.place_cells(s["m"], s["X0"], s["case"]["steps"])
        return {"start": o, "gradient": g, "X": X, "objective": obj}
    if kind == "encoder":
        e = s["enc"]
        loss = e.train(1, lr=1e-3, seed=3)
        mean, logvar = e.predict(1)
        return {"loss": loss.astype(np.float32), "mean": mean.astype(np.float32), "logvar": logvar.astype(np.float32),
                **{k: v.astype(np.float32) for k, v in e.get_params().items()}}
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rc = s["lib"].gpl_kernel_mats_noalloc(s["N"], s["M"], s["Q"], p(s["X"]), p(s["T"]), p(s["rho"]), p(s["Knm"]),
                                          p(s["Kinv"]), p(s["tit"]),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError("gpl_kernel_mats_noalloc: %d" % rc)
    return {"Knm": s["Knm"], "KinvKmn": s["Kinv"], "titsias": s["tit"]}


# ---- the same in float64 with plain torch -----------------------------------------------------------
def _titsias(K, Kmm):
    return (1.0 - (K * torch.cholesky_solve(K.T, torch.linalg.cholesky(Kmm)).T).sum(1)) / 2.0


def _unit_diag(Kmm):
    n = Kmm.shape[0]
    return Kmm * (1.0 - torch.eye(n, device="cuda", dtype=F64)) + torch.eye(n, device="cuda", dtype=F64)


def _prior(w, delta, Kmm):
    """DeltaInv = blockdiag(1/delta_k, Kmm / delta_GP)."""
    d = torch.cat([(1.0 / delta[k]).repeat(n) for k, n in enumerate(w.widths)])
    return torch.block_diag(torch.diag(d), Kmm / delta[-1])


def _dense_counts(w, j):
    y = torch.zeros(w.N, dtype=F64, device="cuda")
    a, b = int(w.ptr_h[j]), int(w.ptr_h[j + 1])
    y[w.cell[a:b].long()] = w.count[a:b]
    return y


class _Irls:
    """W, nu from beta, the Gram, its factor, the coefficient update and phi of one IRLS sweep."""

    def __init__(self, w, beta, sweep):
        w.ptr_h = _np(w.ptr)
        Kmm = _unit_diag(_kernel(w.T, w.T, w.rho))
        K = _kernel(w.X, w.T, w.rho)
        self.Z = torch.cat([w.C, K], 1)
        self.tit = _titsias(K, Kmm)
        self.tt = WT * w.delta[-1] * self.tit
        self.prior = _prior(w, w.delta, Kmm)
        N, J, P = w.N, w.J, w.P
        eta = beta.T @ self.Z.T  # J x N
        W = torch.exp(eta) * (w.s * torch.exp(self.tt))[None, :]
        nu = eta - 1.0
        gene = torch.repeat_interleave(torch.arange(J, device="cuda"), w.ptr[1:] - w.ptr[:-1])
        cell = w.cell.long()
        nu[gene, cell] += w.count / W[gene, cell]
        lk = -W.sum(1)
        lk.index_add_(0, gene, (torch.log(W[gene, cell]) - self.tt[cell]) * w.count)
        self.W, self.nu, self.likelihood = W, nu, lk.sum()
        wr = W / w.Omega[None, :]
        self.b = (wr * nu) @ self.Z  # J x P
        self.Psi = torch.empty(J, P, P, dtype=F64, device="cuda")
        for j in range(J):
            self.Psi[j] = (self.Z * wr[j][:, None]).T @ self.Z + self.prior
        self.L = torch.linalg.cholesky(self.Psi)
        x = torch.cholesky_solve(self.b[:, :, None], self.L)[:, :, 0]
        r = 1.0 if sweep > 100 else (sweep + 1) / 100.0
        self.beta = beta.T * (1 - r) + x * r  # J x P
        quad = (nu * nu * wr).sum(1)
        fit = ((self.L.transpose(1, 2) @ self.beta[:, :, None])[:, :, 0] ** 2).sum(1)
        ph = (quad - fit) / N
        self.phi = torch.clamp(torch.where((ph < 0.0) | torch.isnan(ph), 1.0, ph), 0.01, 1000.0)


def _exact_evaluate(w, st, moved):
    Om, delta, X, T, rho = [t.clone() for t in moved]
    N, J, P, M = w.N, w.J, w.P, w.M
    leaves = [t.requires_grad_(True) for t in (delta, X, T, rho)]
    Kmm = _unit_diag(_kernel(T, T, rho))
    K = _kernel(X, T, rho)
    Z = torch.cat([w.C, K], 1)
    prior = _prior(w, delta, Kmm)
    tit = _titsias(K, Kmm)
    obj = 0.0
    gZ, gD, gO = torch.zeros(N, P, dtype=F64, device="cuda"), torch.zeros(P, P, dtype=F64, device="cuda"), torch.zeros(N, dtype=F64, device="cuda")
    z, pr = Z.detach(), prior.detach()
    Lp = torch.linalg.cholesky(pr)
    ldp = torch.log(torch.diagonal(Lp)).sum()
    step = max(1, min(J, 400_000_000 // (P * P * 8)))
    for j0 in range(0, J, step):
        js = range(j0, min(J, j0 + step))
        wr = st.W[js.start:js.stop] / Om[None, :]
        nu, ph = st.nu[js.start:js.stop], st.phi[js.start:js.stop]
        b = (wr * nu) @ z
        Psi = torch.stack([(z * wr[k][:, None]).T @ z for k in range(len(js))]) + pr
        L = torch.linalg.cholesky(Psi)
        x = torch.cholesky_solve(b[:, :, None], L)[:, :, 0]
        obj = obj + (-0.5 * N * torch.log(ph) + 0.5 * torch.log(wr).sum(1) + ldp
                     - torch.log(torch.diagonal(L, dim1=1, dim2=2)).sum(1) - 0.5 * (nu * nu * wr).sum(1) / ph
                     + 0.5 * (b * x).sum(1) / ph).sum()
        G = -0.5 * torch.cholesky_inverse(L) - 0.5 * (x[:, :, None] * x[:, None, :]) / ph[:, None, None]
        gD += G.sum(0)
        for k in range(len(js)):
            zG = z @ G[k]
            zx = z @ x[k] / ph[k]
            gZ += 2.0 * wr[k][:, None] * zG + torch.outer(wr[k] * nu[k], x[k] / ph[k])
            gw = (z * zG).sum(1) + nu[k] * zx - 0.5 * nu[k] ** 2 / ph[k]
            gO -= wr[k] * gw + 0.5
    gD += 0.5 * J * torch.cholesky_inverse(Lp)
    oinvt = st.W.sum(0) / Om
    extra = -(WT * delta[-1] * oinvt * tit).sum()
    obj = obj + extra.detach() - (IGB / Om + IGA * torch.log(Om)).sum()
    gO += (WT * delta[-1] * oinvt * tit).detach() + IGB / Om - IGA
    (extra + (Z * gZ).sum() + (prior * gD).sum()).backward()
    gd, gX, gT, gr = [t.grad for t in leaves]
    return obj, [gO, gd * delta.detach(), gX, gT, gr * rho.detach()]


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("fit", "de", "encoder"):  # iterations whose every step is rounded
        return None
    with torch.no_grad():
        if kind == "kernels":
            s = prepare(c, seed)
            K = _kernel(s["X"].T, s["T"].T, s["rho"])
            Y = torch.cholesky_solve(K.T, torch.linalg.cholesky(_unit_diag(_kernel(s["T"].T, s["T"].T, s["rho"]))))
            return {"Knm": K.T.contiguous(), "KinvKmn": Y, "titsias": (1.0 - (K * Y.T).sum(1)) / 2.0}
        w = _World(c, seed)
        w.ptr_h = _np(w.ptr)
        if kind == "irls":
            K = _kernel(w.X, w.T, w.rho)
            Z = torch.cat([w.C, K], 1)
            L = torch.linalg.cholesky(Z.T @ Z + _prior(w, w.delta, _unit_diag(_kernel(w.T, w.T, w.rho))))
            y0 = torch.log(0.05 / w.s)[None, :].repeat(w.J, 1)
            gene = torch.repeat_interleave(torch.arange(w.J, device="cuda"), w.ptr[1:] - w.ptr[:-1])
            cell = w.cell.long()
            y0[gene, cell] = torch.log((w.count + 0.05) / w.s[cell])
            st = _Irls(w, torch.cholesky_solve((y0 @ Z).T, L), c["sweep"])
            return {"likelihood": st.likelihood, "beta": st.beta.reshape(-1), "phi": st.phi}
        if kind == "place":
            X0 = w.X + 0.3 * w.rn(w.N, w.Q)
            Kmm = _unit_diag(_kernel(w.T, w.T, w.rho))
            o, g = torch.zeros(w.N, dtype=F64, device="cuda"), None
            lgam, ysum = torch.zeros_like(o), torch.zeros_like(o)
            cell = w.cell.long()
            lgam.index_add_(0, cell, torch.lgamma(w.count + 1.0))
            ysum.index_add_(0, cell, w.count * torch.log(w.s)[cell])
            X = X0.clone()
            with torch.enable_grad():
                X.requires_grad_(True)
                K = _kernel(X, w.T, w.rho)
                tt = WT * w.delta[-1] * _titsias(K, Kmm)
                Kd, td = K.detach().requires_grad_(True), tt.detach().requires_grad_(True)
                step = max(1, 20_000_000 // w.N)
                for j0 in range(0, w.J, step):
                    j1 = min(w.J, j0 + step)
                    y = torch.stack([_dense_counts(w, j) for j in range(j0, j1)], 1)
                    eta = torch.cat([w.C, Kd], 1) @ w.beta[:, j0:j1]
                    part = (y * eta - torch.exp(eta) * (w.s * torch.exp(td))[:, None]).sum(1)
                    part.sum().backward()
                    o += part.detach()
                prior = (X[:, 1:] ** 2).sum(1) / 2.0
                ((K * Kd.grad).sum() + (tt * td.grad).sum() - prior.sum()).backward()
            return {"start": o + ysum - lgam - prior.detach(), "gradient": X.grad, "X": None, "objective": None}
        st = _Irls(w, w.beta, 0)
        if kind == "evaluate":
            moved = w.moved()
            st.Psi = st.L = None
            with torch.enable_grad():
                obj, g = _exact_evaluate(w, st, moved)
            return {"objective": obj, "gradient": torch.cat([t.T.reshape(-1) if t.dim() == 2 else t for t in g])}
        G = torch.randint(0, 3, (c["columns"], w.N), generator=w.g, device="cuda").double()
        dos = torch.randint(0, 3, (c["donors"], w.J, c["variants"]), generator=w.g, device="cuda").double()
        wr = st.W / w.Omega[None, :]
        res = torch.zeros_like(wr)
        for j in range(w.J):
            res[j] = (_dense_counts(w, j) - st.W[j]) / w.Omega
        S = torch.empty(w.J, c["columns"], dtype=F64, device="cuda")
        for l in range(c["columns"]):
            t = (wr * G[l][None, :]) @ st.Z
            u = torch.linalg.solve_triangular(st.L, t[:, :, None], upper=False)[:, :, 0]
            S[:, l] = (res @ G[l]) / torch.sqrt(st.phi * ((wr @ (G[l] ** 2)) - (u * u).sum(1)))
        cis = torch.empty(w.J, c["variants"], dtype=F64, device="cuda")
        for j in range(w.J):
            g = dos[w.donor, j, :]  # N x V
            t = st.Z.T @ (wr[j][:, None] * g)
            u = torch.linalg.solve_triangular(st.L[j], t, upper=False)
            v = (wr[j][:, None] * g * g).sum(0) - (u * u).sum(0)
            cis[j] = (res[j] @ g) / torch.sqrt(st.phi[j] * v)
        return {"S": S, "cis": cis, "LR": cis * cis}
