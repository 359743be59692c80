"""Infinite activations in the warm-start network: an infinity reaches the outputs that
it reaches in FP32 arithmetic, as an infinity, and no others.

Two components that share no edge; node 0 (the first variable, in one component) has
an infinite feature.  Weights, edges and biases are positive, so nothing cancels: a
value is infinite exactly where a path leads to it from node 0.
"""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300.gnn import WarmStartGNN
from oracle import gnn_ref


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [64, 32])
@pytest.mark.parametrize("n,m,density,L", [(40, 6, 0.6, 1), (150, 9, 0.5, 2), (400, 4, 1.0, 2), (60, 90, 0.05, 3)])
def test_infinite_feature(n, m, density, L, hidden):
    rng = np.random.default_rng(n)
    block = lambda s: sp.random(m, n, density=density, random_state=s, format="csr")     # noqa: E731
    A = sp.block_diag([block(1), block(2)]).tocsr()
    A.data = rng.random(A.nnz) + 0.5
    k = m // 2
    p = sps.Problem(c=rng.random(2 * n), A_ub=A[:k], b_ub=rng.random(k), A_eq=A[k:], b_eq=rng.random(2 * m - k),
                    lb=np.zeros(2 * n), ub=np.full(2 * n, np.inf), integer_mask=np.zeros(2 * n, bool))
    with WarmStartGNN(p, hidden=hidden, layers=L, seed=1, max_batch=2, lp_features=False) as net:
        params = (0.01 + 0.02 * rng.random(net.num_params)).astype(np.float32)
        net.set_params(params)
        fvs = [rng.random((2 * n, 4)).astype(np.float32) for _ in range(2)]
        fcs = [rng.random((2 * m, 4)).astype(np.float32) for _ in range(2)]
        fvs[0][0, 1] = np.inf
        X, Y, Lw = net.predict_features(fvs, fcs)
        lay = gnn_ref.Layout(hidden, L, 4, 4)
        for s in range(2):
            x, y, lw = gnn_ref.predict(params, lay, net._ptr, net._idx, net._val, fvs[s], fcs[s])
            assert np.isinf(x[0]) == (s == 0) and np.isfinite(x[n:]).all() and np.isfinite(y[m:]).all()
            np.testing.assert_allclose(X[s], x, rtol=1e-4)             # infinities have to agree
            np.testing.assert_allclose(Y[s], y, rtol=1e-4)
            np.testing.assert_allclose(Lw[s], lw, rtol=1e-4)
