"""The oracle at sizes where the pair products run in integer arithmetic (option pair_form), and the model
comparison, whose products do not, beyond the golden tables' sizes."""
import numpy as np
import pytest

from gaspacho2_b200 import de, synth
from gaspacho2_b200.model import GPLVM
from oracle import port
from tests import golden_util as gu
from tests.test_gpu_parity import _sensitivity

pytestmark = pytest.mark.gpu


def test_phases_in_integer_arithmetic():
    """GLM initialisation, IRLS, objective, gradient and an L-BFGS step; each buffer within 20 times the
    oracle's own rounding sensitivity, 1e-8 at least."""
    ds = synth.make(1, 13, N=3001, G=301)
    ref, sens = _sensitivity(ds, seeds=(0,))
    with GPLVM.from_dataset(ds) as m:
        out = gu.run_phases(m, ds)
        assert m.get_option("pair_form") == 3
    assert int(out["irls_n"]) == int(ref["irls_n"])
    bad = []
    for k, v in out.items():
        if k == "irls_n":
            continue
        e = gu.rel_err(np.atleast_1d(v), np.atleast_1d(ref[k]))
        tol = max(1e-8, 20.0 * sens[k])
        if k in ("obj0", "obj1", "sweep0_lkhd"):
            tol = min(tol, 1e-6)
        if not e <= tol:
            bad.append(f"{k}: {e:.2e} > {tol:.2e}")
    assert not bad, "; ".join(bad)


def test_model_comparison_beyond_the_golden_sizes():
    """1,001 cells x 49 genes at the driver's first two sweeps, where no gene has overshot yet: the bars of the
    golden tables (1e-8 of the largest entry)."""
    ds = synth.make(1, 3, N=1001, G=49, M=12, Q=3, init=True)
    bfs, sweeps, beta, phi = port.de_bfs(ds, ds.init, 5, ds.M, 2)
    out = de.de_bfs(ds.y, ds.z, ds.ls, ds.init, ds.Q, 5, ds.M, 2)
    out.pop("full").close()
    assert out["sweeps"] == sweeps
    assert gu.rel_err(out["BFs"], bfs) <= 1e-8 and gu.rel_err(out["phi"], phi) <= 1e-8


# a gene whose weights overflow, in one range of cells and in several (the flag rises after the first ranges
# have written): the gradient is not finite where the FP64 form's is not, and the same elsewhere
@pytest.mark.parametrize("cells", [0, 512])
def test_non_finite_gene_in_the_gradient(cells):
    ds = synth.make(0, 5, N=2500, G=600, M=64, Q=5, init=False)
    ds.init.rho[:] = 3.0
    out = []
    for c in (cells, 128):
        with GPLVM.from_dataset(ds) as m:
            m.set_option("pair_range_cells", c)
            m.set_params(ds.init)
            beta = 0.2 * np.random.default_rng(3).standard_normal((m.P, 600))
            beta[0, 5] = 800.0
            m.set_beta(beta)
            m.kernel_mats()
            m.expand_delta()
            m.irls_sweep(0, 0)
            m.objective(0, 1)
            out.append(np.concatenate([m.gradient(), m.get("C1")]))
            assert m.get_option("pair_form") == (0 if c == 128 else 3)
    a, b = out
    assert not np.all(np.isfinite(b))
    f = np.isfinite(b)
    assert np.array_equal(np.isfinite(a), f)
    assert np.linalg.norm(a[f] - b[f]) <= 1e-10 * np.linalg.norm(b[f])
