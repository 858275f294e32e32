"""The shared sums and split products at the sizes where their splits change, against NumPy: per-cell
sums over genes, group sums in runs, HK and C2 in ranges, the likelihoods' log products."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


def _evaluate(ds, beta_scale):
    """W and nu from given coefficients, then the objective and gradient; returns what the checks need."""
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        m.kernel_mats()
        m.expand_delta()
        rng = np.random.default_rng(1)
        m.set_beta(beta_scale * rng.standard_normal((m.P, m.J)) - np.eye(m.P, 1) * 1.5)
        m.irls_sweep(0, 0)
        v, g = m.evaluate(m.params_vector())
        out = {k: m.get(k) for k in ("W", "Nu", "C2", "KinvKmn", "tBeta", "phi", "PsiInv", "Kmm", "Kinv", "lkhds",
                                     "DeltaInv", "Dm")}
        return out, (m.N, m.J, m.M, m.P, m.p), v, g.copy()


# cells and genes where the blocks' splits change (1 / several parts, odd remainders), few and many
# dense columns (row tiles of 16, 48, 80 and 144), two variables and one
@pytest.mark.parametrize("config,N,G,M,Q", [(0, 333, 7, 3, 3), (0, 2001, 130, 32, 5), (1, 4097, 65, 60, 5),
                                            (1, 1000, 700, 12, 5), (2, 1900, 40, 150, 10)])
def test_sums_against_numpy(config, N, G, M, Q):
    ds = synth.make(config, 9, N=N, G=G, M=M, Q=Q, init=False)
    ds.init.rho[:] = 2.0
    ds.init.Omega[:] = np.exp(0.2 * np.random.default_rng(2).standard_normal(N))
    o, (N, J, M, P, p), v, g = _evaluate(ds, 0.05)
    om, delta = ds.init.Omega, ds.init.delta
    W = o["W"].reshape(J + 1, N)
    nu = o["Nu"].reshape(J, N)
    oinvt = W[:J].sum(0) / om
    # a sum of n terms in any order: n u of the terms' magnitudes
    assert np.allclose(W[J], oinvt, rtol=2 * J * 2.0 ** -53, atol=0)
    tB = o["tBeta"].reshape(J, P)[:, P - M:]
    Y = o["KinvKmn"].reshape(N, M)
    S = o["PsiInv"].reshape(J, P, P)[:, P - M:, P - M:]
    K = np.triu(o["Kmm"].reshape(M, M).T)
    K = K + np.triu(K, 1).T
    L = np.tril(o["Kinv"].reshape(M, M).T)
    inv = np.linalg.inv(L @ L.T)
    d = delta[-1]
    s1, s2, s3 = (Y * oinvt[:, None]).T @ Y, (tB / o["phi"][:, None]).T @ tB, S.sum(0)
    C2 = (-0.1 * d * s1 / 2 - s2 / d / 2 - s3 / d / 2 + J * inv / 2) * K
    scale = (0.1 * d * np.abs(s1) + np.abs(s2) / d + np.abs(s3) / d + J * np.abs(inv)) / 2
    # C2's terms cancel: the sums' n u and the inverse's M u cond, against the terms' magnitudes
    tol = ((N + J) * 2.0 ** -53 + 100 * M * 2.0 ** -53 * np.linalg.cond(K)) * scale.max()
    assert np.abs(o["C2"].reshape(M, M).T - C2).max() <= tol
    # per-gene likelihoods: l_j without its matrix terms, which enter the same way in every gene's check
    LD = np.diag(o["DeltaInv"].reshape(P, P).T)
    D = o["Dm"].reshape(-1, N)
    assert np.all(np.isfinite(o["lkhds"])) and np.isfinite(v) and np.all(np.isfinite(g)) and LD.size == P and D.size
    a = -0.5 * np.log(om[None, :] / W[:J]).sum(1) - 0.5 * (nu ** 2 * W[:J] / om).sum(1) / o["phi"]
    a -= 0.5 * N * np.log(o["phi"])
    rest = o["lkhds"] - a  # log determinants and the quadratic form
    Z = _model_matrix(ds, D, M, P)
    prior = np.linalg.inv(_prior_inverse(ds, K, delta))
    for j in (0, J // 2, J - 1):
        w = W[j] / om
        psi = (Z * w[:, None]).T @ Z + np.linalg.inv(prior)
        b = Z.T @ (w * nu[j])
        r = -0.5 * np.linalg.slogdet(psi)[1] - 0.5 * np.linalg.slogdet(prior)[1]
        r += 0.5 * b @ np.linalg.solve(psi, b) / o["phi"][j]
        # three sums of N or P terms that nearly cancel: relative to their size
        size = abs(a[j]) + 0.5 * (nu[j] ** 2 * w).sum() / o["phi"][j] + abs(r)
        assert abs(rest[j] - r) <= 1e-11 * size


def _prior_inverse(ds, K, delta):
    z = ds.z
    diag = [1.0 / delta[0]]
    for k in range(z.n_var):
        diag += [1.0 / delta[k + 1]] * int(z.c[k] * z.v[k])
    n, M = len(diag), K.shape[0]
    out = np.zeros((n + M, n + M))
    out[np.arange(n), np.arange(n)] = diag
    out[n:, n:] = K / delta[-1]
    return out


def _model_matrix(ds, D, M, P):
    z, N = ds.z, ds.N
    cols = [np.ones((N, 1))]
    for k in range(z.n_var):
        c = z.columns[k]
        cols.append(np.eye(int(z.c[k]))[np.asarray(c)] if z.c[k] > 1 else np.asarray(c).reshape(N, -1))
    cols.append(D[-M:].T)
    Z = np.concatenate(cols, 1)
    assert Z.shape[1] == P
    return Z
