"""The factorizations and substitutions at the edges of their blocks: the batched Cholesky beyond the
single-panel kernel's range (k_potrf_rows), the kernel matrices' blocked substitution (k_kmm_solve) and
the prior's block factor (k_chol_exact) against NumPy."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _dataset(N, G, M, Q=10, config=0, seed=3):
    ds = synth.make(config, seed, N=N, G=G, M=M, Q=Q, init=False)
    ds.init.rho[:] = 3.0
    return ds


# P = M + 4: just past the panel kernel's 288, whole and broken 32-column panels and 128-row blocks,
# odd (8-byte copies) and even
@pytest.mark.parametrize("M", [285, 316, 317, 380, 413])
def test_cholesky_beyond_one_panel(M):
    ds = _dataset(900, 5, M)
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        P, J = m.P, m.J
        assert P == M + 4
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 0)
        L = np.tril(m.get("Psi").reshape(J, P, P).transpose(0, 2, 1))
        m.gram()
        psi = m.get("Psi").reshape(J, P, P)
    for j in range(J):
        d = np.sqrt(np.diag(psi[j]))
        # backward error of a Cholesky factor: (P + 1) u |L| |L|^T entrywise, at most sqrt(d_a d_b) each
        assert np.all(np.abs(L[j] @ L[j].T - psi[j]) <= 2 * (P + 1) * U * np.outer(d, d))


@pytest.mark.parametrize("N,M,Q", [(1, 1, 2), (127, 31, 5), (128, 32, 5), (129, 33, 5), (1000, 100, 10), (333, 257, 10)])
def test_kernel_substitution(N, M, Q):
    ds = _dataset(max(N, 300), 3, M, Q) if M <= 300 else None
    with GPLVM.from_dataset(synth.cell_subset(ds, np.arange(N), init=False)) as m:
        m.set_params(synth.default_params(N, 3, m.p, M, Q, ds.X0[:N], ds.init.T))
        m.kernel_mats()
        K = m.get("Knm").reshape(M, N).T
        Kmm = np.triu(m.get("Kmm").reshape(M, M).T)
        Y = m.get("KinvKmn").reshape(N, M)
        t = m.get("titsias")
    Kmm = Kmm + np.triu(Kmm, 1).T
    # residual of a backward stable substitution with a Cholesky factor: 3 M u |K| |y| (twice that,
    # for the factor's own error)
    res = np.abs(K - Y @ Kmm)
    assert np.all(res <= 8 * (M + 1) * U * (np.abs(Y) @ np.abs(Kmm) + np.abs(K)) * max(1.0, np.sqrt(M)))
    assert np.all(np.abs(t - (1.0 - (K * Y).sum(1)) / 2.0) <= 4 * (M + 2) * U * (1.0 + (np.abs(K) * np.abs(Y)).sum(1)))


@pytest.mark.parametrize("M", [2, 33, 128, 240, 260])
def test_prior_factor(M):
    """After an objective the lower triangle of DeltaInv holds its factor: the square roots of the
    covariates' diagonal, zeros below them, and the GP block's factor."""
    ds = _dataset(600, 3, M, 10, config=1)
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 0)
        m.objective(0, 1)
        P = m.P
        D = m.get("DeltaInv").reshape(P, P).T
        m.expand_delta()
        A = np.triu(m.get("DeltaInv").reshape(P, P).T)
    A = A + np.triu(A, 1).T
    L = np.tril(D)
    g0 = P - M
    assert np.array_equal(np.diag(L)[:g0], np.sqrt(np.diag(A)[:g0]))
    assert np.count_nonzero(np.tril(L, -1)[:, :g0]) == 0
    d = np.sqrt(np.diag(A))
    assert np.all(np.abs(L @ L.T - A) <= 2 * (P + 1) * U * np.outer(d, d))


# P = M + 4 at the edges of the 32-column panels, of the half-size kernel (160) and of the panel kernel
# (288), odd (8-byte copies) and even
@pytest.mark.parametrize("M", [1, 27, 28, 29, 60, 61, 92, 125, 156, 157, 188, 253, 284, 317])
def test_factor_and_inverse(M):
    ds = _dataset(700, 4, M)
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        P, J = m.P, m.J
        assert P == M + 4
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 0)
        m.objective(0, 1)
        L = np.tril(m.get("Psi").reshape(J, P, P).transpose(0, 2, 1))
        m.gradient()
        X = m.get("PsiInv").reshape(J, P, P)
    for j in range(J):
        # with V = L^-1 (1 + E), |E| <= 2 (P + 2) u |L||V| (its diagonal blocks' inverses included) and
        # X = fl(V^T V): L L^T X - 1 is at most, to first order, 8 (P + 2) u |L||L^T||V^T||L^T||V^T||V|
        V = np.linalg.inv(L[j])
        aL, aV = np.abs(L[j]), np.abs(V)
        bound = aL @ (aL.T @ aV.T @ aL.T @ aV.T) @ aV
        assert np.array_equal(X[j], X[j].T)
        assert np.all(np.abs(L[j] @ (L[j].T @ X[j]) - np.eye(P)) <= 8 * (P + 2) * U * bound)


# the last gene count of the fused tail (one gene per resident CTA) and the first of the separate kernels
@pytest.mark.parametrize("J", [296, 297])
def test_tail_rule_same_bits(J):
    out = []
    for fused in (0, 1):
        ds = _dataset(400, J, 9, 5)
        with GPLVM.from_dataset(ds) as m:
            m.set_option("fused_tail", fused)
            m.set_params(ds.init)
            m.kernel_mats()
            m.glm_init()
            m.irls_sweep(0, 0)
            out.append({k: m.get(k) for k in ("Beta", "phi", "Psi", "lkhds")})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k], equal_nan=True), k


# the first column of a panel is the root of its pivot and the entries times the root's reciprocal, both
# rounded correctly: P = M + 4 in the half-size panel kernel, the panel kernel and the row-block kernel
@pytest.mark.parametrize("M,J", [(9, 2000), (170, 300), (300, 100)])
def test_first_column_rounded_correctly(M, J):
    ds = _dataset(400, J, M)
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        P = m.P
        m.kernel_mats()
        m.glm_init()
        m.irls_sweep(0, 0)
        L = m.get("Psi").reshape(J, P, P).transpose(0, 2, 1)[:, :, 0].copy()
        m.gram()
        psi = m.get("Psi").reshape(J, P, P).transpose(0, 2, 1)[:, :, 0]
    root = np.sqrt(psi[:, 0])
    assert np.array_equal(L[:, 0], root)
    assert np.array_equal(L[:, 1:], psi[:, 1:] * (1.0 / root)[:, None])
