"""More genes than a launch's second dimension counts (65,535): the integer Gram of 65,537 genes through an
IRLS sweep and the objective, against a context of the last hundred of them, which takes the FP64 form."""
import numpy as np
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.formats import Counts, Params
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


def test_more_than_65535_genes():
    N, J, M = 768, 65537, 20
    ds = synth.make(0, 3, N=N, G=3, M=M, Q=2, init=False)
    rng = np.random.default_rng(2)
    i = np.sort(rng.integers(0, N // 2, (J, 2)) + np.array([0, N // 2]), axis=1).astype(np.int32)  # two cells a gene
    x = rng.integers(1, 4, (J, 2)).astype(np.float64)
    out = {}
    for first in (0, J - 100):
        n = J - first
        y = Counts(N, n, i[first:].ravel().copy(), (2 * np.arange(n + 1)).astype(np.int32), x[first:].ravel().copy())
        with GPLVM(y, ds.z, ds.ls, ds.X0, M, 2) as m:
            P = m.P
            beta = 0.3 * np.random.default_rng(4).standard_normal((P, J)) - 1.0
            m.set_params(Params(ds.init.Omega, ds.init.delta, ds.init.X, ds.init.T, ds.init.rho, np.ones(n)))
            m.set_beta(beta[:, first:])
            m.kernel_mats()
            m.expand_delta()
            assert np.isfinite(m.irls_sweep(0, 0))
            m.gram()
            assert (m.get_option("pair_form") & 1) == (first == 0)
            psi = m.get("Psi").reshape(n, P, P)[-100:].copy()
            assert np.isfinite(m.objective(0, 1))
            out[first] = psi
    # 8 times the rms rounding of either form of the dense block, by sqrt(Psi_aa Psi_bb): the integer form's 4 u,
    # the chain's 0.15 sqrt(N) u; the batches' rows, FP64 sums split by the number of genes, lie within that
    u = 2.0 ** -53
    a, b = out[0], out[J - 100]
    d = np.sqrt(np.diagonal(b, axis1=1, axis2=2))
    assert np.all(np.abs(a - b) <= (8 * 4 + 1.2 * np.sqrt(N) + 8) * u * d[:, :, None] * d[:, None, :])
