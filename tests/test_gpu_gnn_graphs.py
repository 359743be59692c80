"""Warm-start network on graphs that are not the transportation family: as many rows as
columns, more rows than columns, long columns, short rows, many rows.  Outputs and
gradient against the FP64 oracle with the tolerances of test_gpu_gnn_shapes; the same
bits whatever the batch; and the time of such a graph against its transpose's."""

import time

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300.gnn import WarmStartGNN
from oracle import gnn_ref
from test_gpu_gnn_shapes import _relu_biases

pytestmark = pytest.mark.gpu


def _graph(m, n, per_row, seed=0):
    rng = np.random.default_rng(seed)
    idx = np.concatenate([rng.choice(n, per_row, replace=False) for _ in range(m)])
    A = sp.csr_matrix((rng.standard_normal(idx.size), idx, np.arange(0, idx.size + 1, per_row)), shape=(m, n))
    k = m // 2
    return sps.Problem(c=rng.random(n), A_ub=A[:k], b_ub=rng.random(k) + 1, A_eq=A[k:], b_eq=rng.random(m - k),
                       lb=np.zeros(n), ub=np.full(n, np.inf), integer_mask=np.zeros(n, bool))


def _inputs(net, B, seed=1):
    rng = np.random.default_rng(seed)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)                             # noqa: E731
    return [f32(net.n, 4) for _ in range(B)], [f32(net.m, 4) for _ in range(B)], \
        [f32(net.n) for _ in range(B)], [f32(net.m) for _ in range(B)], f32(B)


# both sides of the routes: edges per variable against a quarter of the variables per row, 8 edges per variable
@pytest.mark.parametrize("m,n,per_row,B,L", [
    (140, 129, 5, 2, 2), (900, 40, 6, 2, 1), (63, 64, 40, 3, 2), (130, 1040, 16, 1, 2), (130, 1041, 17, 2, 1),
    (20, 256, 100, 2, 3), (127, 128, 8, 1, 2), (127, 128, 7, 1, 2), (1, 300, 300, 2, 1),
])
def test_outputs_and_gradient(m, n, per_row, B, L):
    rng = np.random.default_rng(m + n)
    with WarmStartGNN(_graph(m, n, per_row), layers=L, seed=n, max_batch=B, lp_features=False) as net:
        params = net.params()
        params += 0.1 * rng.standard_normal(params.size).astype(np.float32)
        net.set_params(params)
        lay = gnn_ref.Layout(64, L, 4, 4)
        fvs, fcs, xts, yts, lts = _inputs(net, B)
        X, Y, Lw = net.predict_features(fvs, fcs)
        loss, g = net.loss_grad(fvs, fcs, xts, yts, lts)
    for s in range(B):
        x, y, lw = gnn_ref.predict(params, lay, net._ptr, net._idx, net._val, fvs[s], fcs[s])
        np.testing.assert_allclose(X[s], x, rtol=1e-4, atol=1e-5 * np.abs(x).max())
        np.testing.assert_allclose(Y[s], y, rtol=1e-4, atol=1e-5 * np.abs(y).max())
        assert abs(Lw[s] - lw) <= 1e-4 * (1 + abs(lw))
    (ref_loss, ref_g), (_, up), (_, down) = [
        gnn_ref.loss_grad(params + shift * _relu_biases(lay), lay, net._ptr, net._idx, net._val, fvs, fcs, xts, yts,
                          list(lts), 1.0, 1.0, 0.1, bf16=True) for shift in (0.0, 1e-6, -1e-6)]
    jump = np.abs(up - ref_g) + np.abs(down - ref_g)
    assert abs(loss - ref_loss) <= 1e-5 * (1 + abs(ref_loss))
    assert np.linalg.norm(g - ref_g) <= 1e-4 * np.linalg.norm(ref_g) + np.linalg.norm(jump)


@pytest.mark.parametrize("m,n,per_row", [(500, 4000, 65), (500, 4000, 100), (500, 15000, 70), (500, 12000, 9)])
def test_same_bits_in_every_batch(m, n, per_row):
    """A block or a warp per row, by the rows of the whole batch: an instance's points do not depend on it."""
    B = 34                                                     # 17 000 rows
    with WarmStartGNN(_graph(m, n, per_row), layers=2, seed=3, max_batch=B, lp_features=False) as net:
        fvs, fcs, *_ = _inputs(net, B)
        X, Y, _ = net.predict_features(fvs, fcs)
        for s in (0, 17, B - 1):
            x, y, _ = net.predict_features(fvs[s:s + 1], fcs[s:s + 1])
            assert np.array_equal(x[0], X[s]) and np.array_equal(y[0], Y[s])


@pytest.mark.parametrize("m,n,per_row", [(400, 400, 20), (700, 90, 6), (50, 130, 100)])
def test_outputs_are_as_exact_as_fp32(m, n, per_row):
    """Root mean square error of the points against FP64 at most 7e-7: a value is six rounded sums of
    FP32 (2^-24 each, 1.5e-7 together) of terms that carry the layer's before; a sum whose terms
    are cut to its own last place, 128 of them, is off by more than a part in 10^6."""
    L = 3
    with WarmStartGNN(_graph(m, n, per_row), layers=L, seed=7, max_batch=1, lp_features=False) as net:
        params = net.params()
        fvs, fcs, *_ = _inputs(net, 1)
        X, Y, _ = net.predict_features(fvs, fcs)
        x, y, _ = gnn_ref.predict(params, gnn_ref.Layout(64, L, 4, 4), net._ptr, net._idx, net._val, fvs[0], fcs[0])
    assert np.linalg.norm(X[0] - x) <= 7e-7 * np.linalg.norm(x)
    assert np.linalg.norm(Y[0] - y) <= 7e-7 * np.linalg.norm(y)


def test_many_rows_and_long_columns_keep_pace():
    """40 000 rows of 20 edges on 500 columns (1600 edges each) against the transpose, the same
    edges and nodes: 2 times its time (with the few rows' form 10 times)."""
    def best(p):
        with WarmStartGNN(p, layers=3, seed=1, max_batch=1) as net:
            rng = np.random.default_rng(0)
            f = lambda k: [rng.random((k, 1)).astype(np.float32)]                          # noqa: E731
            fv, fc, xt, yt = f(net.n), f(net.m), [rng.random(net.n)], [rng.random(net.m)]
            calls = (lambda: net.predict_features(fv, fc),
                     lambda: net.loss_grad(fv, fc, xt, yt, np.zeros(1, np.float32)))
            out = []
            for call in calls:
                ts = []
                for _ in range(12):
                    t = time.perf_counter()
                    call()
                    ts.append(time.perf_counter() - t)
                out.append(min(ts[3:]))
            return np.array(out)
    p = _graph(40_000, 500, 20)
    A = sp.vstack([p.A_ub, p.A_eq]).T.tocsr()
    q = sps.Problem(c=np.ones(40_000), A_ub=A[:250], b_ub=np.ones(250), A_eq=A[250:], b_eq=np.ones(250),
                    lb=np.zeros(40_000), ub=np.ones(40_000), integer_mask=np.zeros(40_000, bool))
    assert (best(p) < 4 * best(q)).all()
