"""The model comparison's sums keep one order: its IRLS is undamped, and a gene that overshoots carries a
rounding difference into the leading digits of the table. ``golden/de_order_*.npz`` hold two data sets and
the tables that this library gave for them while the Gram was one chain of FP64 multiply-adds per entry, the
group sums and the products over the cells were unsplit and the kernel solve went row by row: (a) 1,203
cells x 40 genes, Q = 10, M = 40; (b) 1,301 cells x 33 genes with 150 donors, M = 143, beyond the widths
where the split products (144 dense columns) and the panel Cholesky (288) end. The same operations in the same
order give the same bits."""
import os

import numpy as np
import pytest

from gaspacho2_b200 import de, synth
from gaspacho2_b200.formats import Counts, Design, Params
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _load(name):
    z = np.load(os.path.join(GOLDEN, f"de_order_{name}.npz"))
    N, J, M, Q, reduced, sweeps = (int(v) for v in z["dims"])
    y = Counts(N, J, z["cell"].astype(np.int32), z["ptr"].astype(np.int32), z["count"].astype(np.float64))
    lev = [int(z["batch"].max()) + 1] + [1] * z["numeric"].shape[1]
    cols = [z["batch"].astype(np.int32)] + [z["numeric"][:, k:k + 1].copy() for k in range(z["numeric"].shape[1])]
    if z["donor"].size:
        lev.append(150)
        cols.append(z["donor"].astype(np.int32))
    d = Design(N, np.array(lev, np.int32), np.ones(len(lev), np.int32), cols)
    p = Params(z["Omega"], z["delta"], z["X"], z["T"], z["rho"], np.ones(J))
    return z, y, d, p, (Q, reduced, M, sweeps)


@pytest.mark.parametrize("name", ["a", "b"])
def test_table_keeps_its_order(name):
    z, y, d, p, (Q, reduced, M, sweeps) = _load(name)
    ctx = de.open_contexts(y, d, z["s"], z["X"], Q, reduced, M)
    try:
        r = de.de_bfs(y, d, z["s"], p, Q, reduced, M, jtr_max=sweeps, contexts=ctx)
    finally:
        for m in ctx:
            m.close()
    assert np.array_equal(r["BFs"], z["BFs"])
    assert np.array_equal(r["phi"], z["phi"])


def test_kernel_matrices_of_a_selected_model():
    """Forming the kernel matrices again by gpl_kernel_mats keeps the order too (M = 40, beyond the sizes whose
    substitution has the reference's order anyway)."""
    z, y, d, p, (Q, reduced, M, sweeps) = _load("a")
    with GPLVM(y, d, z["s"], z["X"], M, Q) as m:
        m.set_params(p)
        m.de_model("full")
        t, k = m.get("titsias"), m.get("KinvKmn")
        m.kernel_mats()
        assert np.array_equal(m.get("titsias"), t) and np.array_equal(m.get("KinvKmn"), k)


def test_gram_tiles_give_the_same_bits():
    """4,656 pairs x 512, 100 and 40 genes take the Gram's three tile sizes (128 x 128, 64 x 64, 64 x 16): an
    entry is the same chain of multiply-adds in each. 128 cells per range select the FP64 form."""
    ds = synth.make(0, 3, N=600, G=512, M=94, Q=10, init=False)
    ds.init.rho[:] = 3.0
    rng = np.random.default_rng(1)
    beta = 0.1 * rng.standard_normal((98, 512)) - 0.5
    psi = {}
    for J in (512, 100, 40):
        n = int(ds.y.p[J])
        y = Counts(600, J, ds.y.i[:n].copy(), ds.y.p[:J + 1].copy(), ds.y.x[:n].copy())
        with GPLVM(y, ds.z, ds.ls, ds.X0, 94, 10) as m:
            m.set_option("pair_range_cells", 128)
            m.set_params(Params(ds.init.Omega, ds.init.delta, ds.init.X, ds.init.T, ds.init.rho, np.ones(J)))
            assert m.n_dense() == 96 and m.P == 98
            m.set_beta(beta[:, :J])
            m.kernel_mats()
            m.expand_delta()
            m.irls_sweep(0, 0)
            m.gram()
            psi[J] = m.get("Psi").reshape(J, -1)
    assert np.array_equal(psi[40], psi[512][:40])
    assert np.array_equal(psi[100], psi[512][:100])
