"""The column-pair products in integer arithmetic modulo fourteen moduli (k_crt.cu) on the GPU: the
Gram against extended precision, both products against the DMMA form (pair_range_cells below a tile
of the integer form selects it), and operands that are not finite."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


def _context(ds, cells=0):
    m = GPLVM.from_dataset(ds)
    m.set_option("pair_range_cells", cells)
    m.set_params(ds.init)
    m.kernel_mats()
    m.glm_init()
    m.irls_sweep(0, 0)
    return m


def _dataset(N, G, M, Q=10, config=2, seed=5):
    ds = synth.make(config, seed, N=N, G=G, M=M, Q=Q, init=False)
    ds.init.rho[:] = 3.0
    ds.init.Omega[:] = np.exp(0.3 * np.random.default_rng(seed).standard_normal(N))
    return ds


# cells: below, at and past K chunks of 128; genes and pairs around the 256-wide tiles; one range of
# cells, several, and a last one of a single cell
@pytest.mark.parametrize("N,G,M,cells", [(1664, 64, 90, 0), (1665, 255, 60, 0), (2000, 257, 52, 0),
                                         (4097, 256, 40, 1024), (3000, 300, 128, 512)])
def test_gram_against_extended_precision(N, G, M, cells):
    ds = _dataset(N, G, M)
    with _context(ds, cells) as m:
        m.expand_delta()
        m.gram()
        P, nd = m.P, m.n_dense()
        assert N * G * nd * (nd + 1) // 2 >= 4e8  # the integer form's range
        psi = m.get("Psi").reshape(G, P, P)
        W = m.get("W").reshape(-1, N)
        D = m.get("Dm").reshape(nd, N).astype(np.longdouble)
        prior = m.get("DeltaInv").reshape(P, P).T
        cols = np.array([0] + list(range(5, 8)) + list(range(P - M, P)))
    om = ds.init.Omega.astype(np.longdouble)
    prior = np.triu(prior) + np.triu(prior, 1).T
    for j in (0, 1, G // 2, G - 1):
        w = W[j].astype(np.longdouble)
        ref = (D * (w / om)) @ D.T
        # Entry (a, b) is the product of rows A = D_a D_b / Omega and w. Scaled norms lie in (R/2, R],
        # R = 2^54.6, so rounding K entries by at most 1/2 moves a row by sqrt(K) / R of its norm at
        # most; the products, the value and the sum with the prior round a few times at 2^-53.
        sq = (D / om) ** 2 @ (D ** 2).T
        bound = (2.0 * np.sqrt(N) * 2.0 ** -54.6 + 2.0 ** -52) * np.sqrt(sq * (w @ w))
        bound = bound + 2.0 ** -50 * (np.abs(ref) + np.abs(prior[np.ix_(cols, cols)]))
        err = np.abs(psi[j][np.ix_(cols, cols)] - ref - prior[np.ix_(cols, cols)])
        assert np.all(err <= bound), float((err / bound).max())
        # rms error, relative to the diagonal, below the DMMA form's 1e-15 at these sizes
        d = np.sqrt(np.diag(ref))
        assert float(np.sqrt(np.mean((err / np.outer(d, d)) ** 2))) < 1e-15


@pytest.mark.parametrize("config,N,G,M,Q", [(0, 2001, 400, 32, 3), (1, 3000, 201, 64, 5), (2, 2500, 333, 150, 10)])
def test_evaluation_against_dmma_form(config, N, G, M, Q):
    """Objective and gradient in both forms. Their Psi_j differ by some 2^-50 of the diagonal; the
    gradient carries that times the conditioning of Psi_j (below 1e4 with these length-scales)."""
    ds = _dataset(N, G, M, Q, config)
    out = []
    for cells in (0, 128):
        with _context(ds, cells) as m:
            x = m.params_vector()
            v, g = m.evaluate(x)
            out.append((v, g.copy()))
    assert abs(out[0][0] - out[1][0]) <= 1e-12 * abs(out[1][0])
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-10 * np.linalg.norm(out[1][1])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_operands_take_the_dmma_form(bad):
    """A cell whose 1/Omega is not finite: the integer form stands back and Psi is the DMMA form's,
    non-finite where that is."""
    ds = _dataset(2000, 300, 64)
    psi = []
    for cells in (0, 128):
        with _context(ds, cells) as m:
            ds.init.Omega[7] = 0.0 if np.isinf(bad) else bad
            m.set_params(ds.init)
            m.gram()
            psi.append(m.get("Psi"))
            ds.init.Omega[7] = 1.0
    a, b = psi
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert not np.all(np.isfinite(a))
    f = np.isfinite(a)
    assert np.allclose(a[f], b[f], rtol=1e-12, atol=1e-12 * np.abs(b[f]).max())


# The sums over a cell's pair row, a warp or a block per cell (2,368 cells, 96 and 160 columns), V from
# memory (few genes) and from residues, against ranges of 128 cells, which take the DMMA form and a block
# per cell; and the rules' edges in cells and genes. Tolerances as above.
@pytest.mark.parametrize("N,G,M", [(2368, 40, 94), (2368, 40, 95), (2367, 40, 94), (2368, 40, 158), (2369, 40, 159),
                                   (2368, 600, 94), (2369, 600, 95), (2368, 600, 20), (511, 40, 20), (512, 32, 20),
                                   (513, 31, 21), (520, 1000, 3)])
def test_pair_rows_forms(N, G, M):
    ds = _dataset(N, G, M, 10, 1)
    out = []
    for cells in (0, 128):
        with _context(ds, cells) as m:
            x = m.params_vector()
            v, g = m.evaluate(x)
            out.append((v, g.copy()))
    assert abs(out[0][0] - out[1][0]) <= 1e-12 * abs(out[1][0])
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-10 * np.linalg.norm(out[1][1])
