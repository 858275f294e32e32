"""The integer pair products (k_crt.cu) where the operands' rows spread over many orders of magnitude: their
rounding is relative to a row's norm, so they have to notice where that is more than the FP64 form's."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _share(K):
    return U * max(4.0, 0.1 * np.sqrt(K))


def _context(N, G, M, Q=5, config=0, seed=5):
    ds = synth.make(config, seed, N=N, G=G, M=M, Q=Q, init=False)
    ds.init.rho[:] = 3.0
    ds.init.Omega[:] = np.exp(0.3 * np.random.default_rng(seed).standard_normal(N))
    m = GPLVM.from_dataset(ds)
    m.set_params(ds.init)
    return ds, m


# genes at one scale, and over seven orders of magnitude; one gene with a cell at e^30 of the others
@pytest.mark.parametrize("lo,hi,outlier", [(0.0, 0.0, 0.0), (np.log(1e-4), np.log(1e3), 0.0),
                                           (np.log(1e-4), np.log(1e3), 30.0)])
def test_gradient_pairs_of_genes_far_apart(lo, hi, outlier):
    N, G, M = 2500, 600, 64
    ds, m = _context(N, G, M)
    with m:
        rng = np.random.default_rng(3)
        beta = 0.2 * rng.standard_normal((m.P, G))
        beta[0] = rng.uniform(lo, hi, G)
        if outlier:
            beta[-1, 7] = outlier  # the cells near one inducing point
        m.set_beta(beta)
        m.kernel_mats()
        m.expand_delta()
        m.irls_sweep(0, 0)
        m.objective(0, 1)
        got = []
        for cells in (0, 128):  # 128 cells per range: the FP64 form, on the same factors
            m.set_option("pair_range_cells", cells)
            m.gradient()
            assert m.get_option("pair_form") == (0 if cells else 3)
            got.append(m.get("C1").reshape(M, N))
        W = m.get("W").reshape(-1, N)[:G]
        D = m.get("Dm").reshape(m.n_dense(), N)
        P = m.P
        cols = np.array([0] + list(range(P - D.shape[0] + 1, P)))
        Sd = np.diagonal(m.get("PsiInv").reshape(G, P, P), axis1=1, axis2=2)[:, cols]
    V = (W.T @ Sd) / ds.init.Omega[:, None]  # diagonal pairs, positive
    # U_a = sum_b D_b V_ab, |V_ab| <= sqrt(V_aa V_bb): 8 times the rms rounding of either form (the integer
    # form's share, the chain's 0.15 sqrt(G) u) and the sum over b of both; C1 = (terms common to both - U) D
    size = np.sqrt(V) * (np.abs(D.T) * np.sqrt(V)).sum(1)[:, None]
    tol = (8 * _share(G) + 1.2 * np.sqrt(G) * U + 2 * (D.shape[0] + 4) * U) * size
    K = np.abs(D[-M:])
    err = np.abs(got[0] - got[1])
    assert np.all(err <= K * tol.T[-M:] + 4 * U * (np.abs(got[1]) + K * size.T[-M:])), \
        float((err / (K * size.T[-M:])).max())


def _psi(m, ds, beta):
    m.set_beta(beta)
    m.kernel_mats()
    m.expand_delta()
    m.irls_sweep(0, 0)
    m.gram()
    assert m.get_option("pair_form") & 1
    return m.get("Psi").reshape(m.J, m.P, m.P)


# the log of a gene's weight near one inducing point over the others', the genes that have it of 600 (on the
# list's small and large tiles), cells per range (0: one range)
@pytest.mark.parametrize("spread,n_out,cells", [(6.0, 60, 0), (10.0, 3, 0), (14.0, 60, 0), (14.0, 48, 512), (30.0, 49, 0),
                                                (40.0, 3, 512), (40.0, 600, 0)])
def test_gram_of_spread_weights(spread, n_out, cells):
    N, G, M = 2500, 600, 64
    ds, m = _context(N, G, M, Q=2)
    with m:
        m.set_option("pair_range_cells", cells)
        ds.init.rho[:] = 0.2  # columns of few cells each
        m.set_params(ds.init)
        beta = 0.2 * np.random.default_rng(3).standard_normal((m.P, G))
        for j in range(n_out):
            beta[m.P - M + j % M, j] = spread
        psi = _psi(m, ds, beta)
        nd, P = m.n_dense(), m.P
        W = m.get("W").reshape(-1, N)[:G]
        D = m.get("Dm").reshape(nd, N).astype(np.longdouble)
        prior = np.triu(m.get("DeltaInv").reshape(P, P).T)
    prior = prior + np.triu(prior, 1).T
    cols = np.array([0] + list(range(P - nd + 1, P)))
    om = ds.init.Omega.astype(np.longdouble)
    # 8 times the rms rounding of either form (the integer form's share, the chain's 0.15 sqrt(N) u) and a few
    # roundings of the entry, by the scale sqrt(Psi_aa Psi_bb) of both
    tol = 8 * _share(N) + 1.2 * np.sqrt(N) * U + 8 * U
    for j in (0, 1, 2, n_out - 1, G // 2, G - 1):
        ref = (D * (W[j].astype(np.longdouble) / om)) @ D.T + prior[np.ix_(cols, cols)]
        d = np.sqrt(np.diag(ref))
        err = np.abs(psi[j][np.ix_(cols, cols)] - ref) / np.outer(d, d)
        assert np.all(err <= tol), (j, float(err.max() / U))


def test_non_finite_gene_leaves_the_others():
    """A gene whose weights overflow takes the FP64 form alone: the others keep their bits."""
    N, G, M = 2500, 600, 64
    ds, m = _context(N, G, M, Q=2)
    with m:
        beta = 0.2 * np.random.default_rng(3).standard_normal((m.P, G))
        a = _psi(m, ds, beta).copy()
        beta[0, 5] = 800.0
        b = _psi(m, ds, beta)
    assert not np.all(np.isfinite(b[5]))
    keep = np.arange(G) != 5
    assert np.all(np.isfinite(b[keep])) and np.array_equal(a[keep], b[keep])


@pytest.mark.parametrize("spread", [0.0, 14.0, 20.0, 23.0])
def test_genotype_columns_of_spread_weights(spread):
    """Columns that are zero where three genes have their mass: in one call (32 columns, the integer form) and
    one by one (the FP64 form). The variance that is left of g^T diag(w) g is at least 1e-3 of it."""
    N, G, M, L = 2500, 600, 64, 32
    ds, m = _context(N, G, M, Q=2)
    with m:
        ds.init.rho[:] = 0.2
        m.set_params(ds.init)
        beta = 0.2 * np.random.default_rng(3).standard_normal((m.P, G))
        beta[m.P - M, [5, 200, 599]] = spread
        m.set_beta(beta)
        m.kernel_mats()
        m.expand_delta()
        m.irls_sweep(0, 0)
        K = m.get("Knm").reshape(M, N)[0]
        geno = np.random.default_rng(7).normal(1.0, 0.7, (N, L)) * (K < 1e-3)[:, None]
        S = m.score_stats(geno)
        one = np.concatenate([m.score_stats(geno[:, k:k + 1]) for k in range(L)], 1)
    assert np.all(np.isfinite(one))
    assert np.all(np.abs(S - one) <= 1e-9 * (1.0 + np.abs(one)))


@pytest.mark.parametrize("N,om", [(20000, 1.423), (60000, 1.2225)])
def test_equal_entries_round_to_nothing_on_average(N, om):
    """Cells that share one Omega: the intercept's row is one value whose nearest integer is off by 45 u and 77 u
    here, and a sum rounded to nearest by as much; a random rounding averages out over the cells. The diagonal
    stays within the share that the form allows itself (14 u and 24 u)."""
    G, M = 300, 30
    ds = synth.make(0, 5, N=N, G=G, M=M, Q=5, init=False)
    ds.init.rho[:] = 3.0
    ds.init.Omega[:] = om
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        psi = _psi(m, ds, 0.2 * np.random.default_rng(3).standard_normal((m.P, G)))
        W = m.get("W").reshape(-1, N)[:G]
        prior = m.get("DeltaInv").reshape(m.P, m.P)[0, 0]
    ref = W.astype(np.longdouble).sum(1) / np.longdouble(om) + prior
    assert np.all(np.abs(psi[:, 0, 0] - ref) <= (_share(N) + 2 * U) * ref)
