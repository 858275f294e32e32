"""More genes than a launch's second dimension counts (65,535): the integer Gram of 65,537 genes through an
IRLS sweep and the objective, against a context of the last hundred of them. A gene's integer sums depend
on its own row alone, so its Psi_j is the same bits."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.formats import Counts, Params
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


def test_more_than_65535_genes():
    N, J, M = 512, 65537, 1
    ds = synth.make(0, 3, N=N, G=3, M=M, Q=2, init=False)
    rng = np.random.default_rng(2)
    i = np.sort(rng.integers(0, N // 2, (J, 2)) + np.array([0, N // 2]), axis=1).astype(np.int32)  # two cells a gene
    x = rng.integers(1, 4, (J, 2)).astype(np.float64)
    out = {}
    for first in (0, J - 100):
        n = J - first
        y = Counts(N, n, i[first:].ravel().copy(), (2 * np.arange(n + 1)).astype(np.int32), x[first:].ravel().copy())
        with GPLVM(y, ds.z, ds.ls, ds.X0, M, 2) as m:
            P, nd = m.P, m.n_dense()
            beta = 0.3 * np.random.default_rng(4).standard_normal((P, J)) - 1.0
            m.set_params(Params(ds.init.Omega, ds.init.delta, ds.init.X, ds.init.T, ds.init.rho, np.ones(n)))
            m.set_beta(beta[:, first:])
            m.kernel_mats()
            m.expand_delta()
            assert np.isfinite(m.irls_sweep(0, 0))
            m.gram()
            assert m.get_option("pair_form") & 1
            psi = m.get("Psi").reshape(n, P, P)[-100:].copy()
            assert np.isfinite(m.objective(0, 1))
            out[first] = psi
    a, b = out[0], out[J - 100]
    dense = [0] + list(range(P - nd + 1, P))  # columns 1, 2: the batches
    assert np.array_equal(a[:, dense][:, :, dense], b[:, dense][:, :, dense])
    # the batches' rows are FP64 sums over the cells, split by the number of genes: each is off by at most
    # N u sum |terms| <= N u sqrt(Psi_aa Psi_bb)
    d = np.sqrt(np.diagonal(b, axis1=1, axis2=2))
    assert np.all(np.abs(a - b) <= 2 * N * 2.0 ** -53 * d[:, :, None] * d[:, None, :])
