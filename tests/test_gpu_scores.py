"""The genotype statistics where their blocks change (variants and columns around 16 and 32, a single
one, several passes), against NumPy at the fitted state."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,N,G,M,L,V,donors", [(2, 1800, 20, 20, 1, 1, True), (2, 2400, 70, 33, 17, 16, True),
                                                     (2, 2000, 9, 150 - 16, 40, 33, True), (0, 1500, 30, 12, 33, 0, False)])
def test_scores_against_numpy(config, N, G, M, L, V, donors):
    ds = synth.make(config, 4, N=N, G=G, M=M, Q=5, init=False)
    ds.init.rho[:] = 2.0
    rng = np.random.default_rng(7)
    ds.init.Omega[:] = np.exp(0.2 * rng.standard_normal(N))
    geno = rng.normal(1.0, 0.7, (N, L))
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 30)
        S = m.score_stats(geno)
        if V:
            nd = int(ds.z.c[-1])
            dos = rng.integers(0, 3, (nd, G, V)).astype(np.int8)
            cis, lr = m.cis_stats(dos, ds.z.n_var - 1)
        W = m.get("W").reshape(-1, N)[:G]
        phi = m.get("phi")
        P = m.P
        Ls = np.tril(m.get("Psi").reshape(G, P, P).transpose(0, 2, 1))
        D = m.get("Dm").reshape(-1, N)
    z = ds.z
    cols = [np.ones((N, 1))]
    for k in range(z.n_var):
        c = z.columns[k]
        cols.append(np.eye(int(z.c[k]))[np.asarray(c)] if z.c[k] > 1 else np.asarray(c).reshape(N, -1))
    Z = np.concatenate(cols + [D[-M:].T], 1)
    om, y = ds.init.Omega, ds.y
    for j in range(0, G, max(1, G // 7)):
        yj = np.zeros(N)
        a, b = int(y.p[j]), int(y.p[j + 1])
        yj[y.i[a:b]] = y.x[a:b]
        w = W[j] / om

        def ref(g):
            u = np.linalg.solve(Ls[j], Z.T @ (w[:, None] * g))
            v = (w[:, None] * g * g).sum(0) - (u * u).sum(0)
            return ((yj - W[j]) / om) @ g / np.sqrt(phi[j] * v), v / (w[:, None] * g * g).sum(0)

        s, kept = ref(geno)
        # the variance is what is left of g^T diag(w) g: its rounding grows by the inverse of that share
        assert np.all(np.abs(S[j] - s) <= 1e-12 * (1.0 + np.abs(s)) / np.minimum(kept, 1.0))
        if V:
            s, kept = ref(dos[np.asarray(z.columns[-1]), j, :].astype(float))
            assert np.all(np.abs(cis[j] - s) <= 1e-10 * (1.0 + np.abs(s)) / np.minimum(kept, 1.0))
            assert np.array_equal(lr[j], cis[j] ** 2)


@pytest.mark.parametrize("N,G,M,L", [(513, 32, 20, 2), (1000, 40, 33, 40), (2400, 257, 8, 33), (3001, 300, 128, 64)])
def test_columns_in_integer_arithmetic(N, G, M, L):
    """Z^T diag(W/Omega) g of the columns by the integer form (one group of columns and several, one range of
    cells) against the DMMA form, which a single column and a column that is not finite take. Both are exact
    to some 2^-50 of the norms; a score's variance is what is left of g^T diag(w) g, here at least 1e-3."""
    ds = synth.make(2, 4, N=N, G=G, M=M, Q=5, init=False)
    ds.init.rho[:] = 2.0
    geno = np.random.default_rng(7).normal(1.0, 0.7, (N, L))
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 30)
        S = m.score_stats(geno)
        one = np.concatenate([m.score_stats(geno[:, k:k + 1]) for k in range(L)], 1)
        geno[5, L - 1] = np.nan
        T = m.score_stats(geno)
    assert np.all(np.isfinite(S))
    assert np.all(np.abs(S - one) <= 1e-9 * (1.0 + np.abs(one)))
    assert np.all(np.isnan(T[:, L - 1]))
    assert np.all(np.abs(T[:, :L - 1] - one[:, :L - 1]) <= 1e-9 * (1.0 + np.abs(one[:, :L - 1])))
