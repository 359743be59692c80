"""Warm-start network at the sizes where its kernels change: tiles of 128 nodes (an
instance smaller than a tile, tiles that hold two instances, a remainder),
constraint rows above and below a block each, nodes without edges, one and several
layers, both widths; forward and gradient against the FP64 oracle with the
tolerances of test_gpu_gnn (FP32 arithmetic over these sizes).  The gradient jumps
where a ReLU's argument is zero to FP32 rounding, and among these sizes' up to
10^5 units some are: what the oracle's own gradient moves by when every bias
moves by that rounding (1e-6 either way) is allowed on top."""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300 import gnn
from sovereign_solver_gb300.gnn import WarmStartGNN
from oracle import gnn_ref

pytestmark = pytest.mark.gpu

SHAPES = [  # variables, rows, density, instances, layers, hidden
    (1, 1, 1.0, 1, 1, 64), (63, 9, 0.2, 5, 2, 64), (127, 5, 0.5, 2, 2, 64), (128, 11, 0.1, 3, 3, 64),
    (129, 140, 0.05, 4, 1, 64), (300, 7, 0.9, 3, 2, 64), (515, 260, 0.004, 2, 3, 64), (1000, 3, 1.0, 4, 4, 64),
    (63, 9, 0.2, 5, 2, 32), (515, 60, 0.2, 2, 3, 32),
]


def _relu_biases(lay):
    """1 at the biases of the ReLU layers."""
    e = np.zeros(lay.size)
    for name, o, shape, _ in lay.items:
        if name[0] == "b" and name[1] in "vc":
            e[o:o + int(np.prod(shape))] = 1.0
    return e


@pytest.mark.parametrize("n,m,density,B,L,H,F", [(*s, (4, 4)) for s in SHAPES]
                         + [(300, 40, 0.06, 3, 2, 64, (3, 5)), (300, 40, 0.06, 3, 2, 64, (8, 1))])
def test_forward_and_gradient_match_oracle(n, m, density, B, L, H, F, monkeypatch):
    monkeypatch.setattr(gnn, "FV", F[0])                 # feature widths of the network's inputs
    monkeypatch.setattr(gnn, "FC", F[1])
    rng = np.random.default_rng(n + m)
    A = sp.random(m, n, density=density, random_state=n, format="csr")
    A.data = rng.standard_normal(A.nnz)
    k = m // 2
    p = sps.Problem(c=rng.random(n), A_ub=A[:k], b_ub=rng.random(k) + 1, A_eq=A[k:], b_eq=rng.random(m - k),
                    lb=np.zeros(n), ub=np.full(n, np.inf), integer_mask=np.zeros(n, bool))
    with WarmStartGNN(p, hidden=H, layers=L, seed=n, max_batch=B, lp_features=False) as net:
        f32 = lambda *s: rng.standard_normal(s).astype(np.float32)                      # noqa: E731
        fvs, fcs = [f32(n, F[0]) for _ in range(B)], [f32(m, F[1]) for _ in range(B)]
        xts, yts, lts = [f32(n) for _ in range(B)], [f32(m) for _ in range(B)], f32(B)
        params = net.params()
        params += 0.1 * f32(params.size)                                                 # biases too
        net.set_params(params)
        lay = gnn_ref.Layout(H, L, *F)
        X, Y, Lw = net.predict_features(fvs, fcs)
        loss, g = net.loss_grad(fvs, fcs, xts, yts, lts)
        loss2, g2 = net.loss_grad(fvs, fcs, xts, yts, lts)
        X2, Y2, _ = net.predict_features(fvs, fcs)
    assert loss == loss2 and np.array_equal(g, g2) and np.array_equal(X, X2) and np.array_equal(Y, Y2)
    for s in range(B):
        x, y, lw = gnn_ref.predict(params, lay, net._ptr, net._idx, net._val, fvs[s], fcs[s])
        np.testing.assert_allclose(X[s], x, rtol=1e-4, atol=1e-5 * np.abs(x).max())
        np.testing.assert_allclose(Y[s], y, rtol=1e-4, atol=1e-5 * np.abs(y).max())
        assert abs(Lw[s] - lw) <= 1e-4 * (1 + abs(lw))
    ref = [gnn_ref.loss_grad(params + shift * _relu_biases(lay), lay, net._ptr, net._idx, net._val, fvs, fcs, xts,
                             yts, list(lts), 1.0, 1.0, 0.1, bf16=True) for shift in (0.0, 1e-6, -1e-6)]
    (ref_loss, ref_g), (_, up), (_, down) = ref
    jump = np.abs(up - ref_g) + np.abs(down - ref_g)
    assert abs(loss - ref_loss) <= 1e-5 * (1 + abs(ref_loss))
    assert np.linalg.norm(g - ref_g) <= 1e-4 * np.linalg.norm(ref_g) + np.linalg.norm(jump)
    for name, o, shape, _ in lay.items:
        q = slice(o, o + int(np.prod(shape)))
        assert np.linalg.norm(g[q] - ref_g[q]) <= 2e-3 * np.linalg.norm(ref_g[q]) + 1e-7 + np.linalg.norm(jump[q]), name
