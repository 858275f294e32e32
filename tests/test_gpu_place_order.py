"""The placement's sums keep one order: a cell's L-BFGS divides by differences of gradients and carries a
rounding some 1e8 times as far, beyond 1e-7 of its coordinates. ``golden/place_order_*.npz`` hold two data sets
and what this library gave for them while every sum was one chain (over the genes for the objective, the
weights and the residuals against the coefficients, over the inducing points for the gradient) and the kernel
solve went row by row: (a) 1,201 cells x 150 genes, Q = 2, M = 14; (b) 703 x 130, Q = 10, M = 40. The same
operations in the same order give the same bits."""
import os

import numpy as np
import pytest

from gaspacho2_b200.encoder import cell_objective, place_cells
from gaspacho2_b200.formats import Counts, Design, Params
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("name", ["a", "b"])
def test_placement_keeps_its_order(name):
    z = np.load(os.path.join(GOLDEN, f"place_order_{name}.npz"))
    N, J, M, Q, steps = (int(v) for v in z["dims"])
    y = Counts(N, J, z["cell"].astype(np.int32), z["ptr"].astype(np.int32), z["count"].astype(np.float64))
    lev = [int(z["batch"].max()) + 1] + [1] * z["numeric"].shape[1]
    cols = [z["batch"].astype(np.int32)] + [z["numeric"][:, k:k + 1].copy() for k in range(z["numeric"].shape[1])]
    d = Design(N, np.array(lev, np.int32), np.ones(len(lev), np.int32), cols)
    with GPLVM(y, d, z["s"], z["Xfit"], M, Q) as m:
        m.set_params(Params(z["Omega"], z["delta"], z["Xfit"], z["T"], z["rho"], np.ones(J)))
        m.set_beta(z["beta"])
        o, g = cell_objective(m, z["X0"], grad=True)
        X, obj, _ = place_cells(m, z["X0"], steps)
    assert np.array_equal(o, z["objective0"]) and np.array_equal(g, z["gradient"])
    assert np.array_equal(X, z["X"]) and np.array_equal(obj, z["objective"])
