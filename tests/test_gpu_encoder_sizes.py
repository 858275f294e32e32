"""The encoder's predictions and batch sums where their tiling can go wrong.

A prediction runs its rows 32,768 at a time in tiles of 128 rows, and the outputs in tiles of 32 of
the 2Q columns; the bias gradients are summed 32 columns and 64 rows at a time. Checked against the
float64 restatement (oracle/encoder_oracle.py), which has the same BF16 rounding points: what may
differ is the FP32 accumulation (relative 256 * 2^-24 = 2e-5) and, by it, now and then the rounding of
a hidden value to its neighbour, 2^-8 of a value below about 4 times a weight below about 4 / sqrt(256):
4e-3 each, so no output may be further off than 1e-2, and the L2 norms than 2e-3.
"""
from types import SimpleNamespace

import numpy as np
import pytest
import scipy.sparse as sp

from gaspacho2_b200.encoder import Encoder
from oracle import encoder_oracle as eo

pytestmark = pytest.mark.gpu


def _cells(N, G, seed):
    rng = np.random.default_rng(seed)
    a = sp.random(N, G, density=0.3, format="csc", random_state=seed)
    a.data = rng.integers(1, 20, a.nnz).astype(np.float64)
    ls = rng.uniform(0.5, 2.0, N)
    y = SimpleNamespace(N=N, J=G, i=a.indices, p=a.indptr, x=a.data)
    return y, ls, np.log1p(a.toarray() / ls[:, None]), rng.permutation(N).astype(np.int32)


@pytest.mark.parametrize("N,n_in,Q", [(1, 5, 1), (127, 128, 16), (129, 130, 17), (32768, 40, 5), (32897, 33, 32)])
def test_predictions_match_oracle(N, n_in, Q):
    first, ls0, F0, o0 = _cells(100, n_in, 3)
    y, ls, F, order = _cells(N, n_in, 4)
    genes = np.arange(n_in)
    with Encoder(n_in, Q, hidden=256, batch=128, seed=5) as enc:
        params = enc.get_params()
        rng = np.random.default_rng(6)
        for b in ("b1", "b2", "b3"):
            params[b] = rng.standard_normal(params[b].shape).astype(np.float32).astype(np.float64)
        enc.set_params(params)
        # a small set first: the buffers then grow for the larger one, and serve the small one again
        enc.set_cells(0, first, ls0, genes, o0)
        enc.set_cells(1, y, ls, genes, order)
        for which, feats in ((0, F0), (1, F), (0, F0)):
            want, _ = eo.forward(params, feats)
            mean, lv = enc.predict(which)
            got = np.concatenate([mean, lv], axis=1)
            assert np.max(np.abs(got - want)) <= 1e-2
            assert np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("batch,Q", [(128, 1), (384, 16), (256, 17), (128, 32)])
def test_batch_sums_match_oracle(batch, Q):
    y, ls, F, order = _cells(batch, 20, 7)
    X = np.random.default_rng(8).standard_normal((batch, Q))
    with Encoder(20, Q, hidden=128, batch=batch, seed=9) as enc:
        enc.set_cells(0, y, ls, np.arange(20), order)
        enc.set_targets(X)
        loss, g = enc.grads(0)
        want, gw, _ = eo.loss_and_grads(enc.get_params(), F[order], X[order])
        assert abs(loss - want) <= 1e-5 * abs(want)
        for k in gw:
            assert g[k].shape == gw[k].shape
            assert np.linalg.norm(g[k] - gw[k]) <= 2e-3 * np.linalg.norm(gw[k]), k
