"""The weight gradient's products of FP32 values in full: nothing of z h is left out.

Two variables with the same activation h and gradients z and -(z without its last eight
bits): their products cancel up to the last bits of z, times all of h.  The parts of the
products add up exactly here, so the sum has no rounding but its own.
"""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300.gnn import WarmStartGNN
from oracle import gnn_ref


def _float(bits):
    return np.uint32(bits).view(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("edges", [0, 2])                     # both routes of the forward pass
@pytest.mark.parametrize("z,h", [(0x3FFFFFFF, 0x3FFFFFFF), (0x3F8000FF, 0x3F80FF01), (0x40ABCDEF, 0x3F123456)])
def test_last_bits_of_a_product(z, h, edges):
    A = sp.csr_matrix(np.ones((1, 2)) if edges else np.zeros((1, 2)))
    p = sps.Problem(c=np.ones(2), A_ub=A, b_ub=np.ones(1), A_eq=sp.csr_matrix((0, 2)), b_eq=np.zeros(0),
                    lb=np.zeros(2), ub=np.ones(2), integer_mask=np.zeros(2, bool))
    lay = gnn_ref.Layout(64, 1, 4, 4)
    P = {name: np.zeros(shape) for name, _, shape, _ in lay.items}
    P["Wv"][:, 0] = 1.0                                       # every activation is the first feature
    P["bv0"][:] = 1.0                                         # every output is 1: nothing is masked
    P["wx"][:2] = (1.0, -1.0)                                 # x0 = 0, and z = x0 - target for output 0
    zs = np.array([_float(z), -_float(z & 0xFFFFFF00)], np.float32)
    fv = np.zeros((2, 4), np.float32)
    fv[:, 0] = _float(h)
    with WarmStartGNN(p, layers=1, seed=0, max_batch=1, lp_features=False) as net:
        net.set_params(lay.pack(P).astype(np.float32))
        x, _, _ = net.predict_features([fv], [np.zeros((1, 4), np.float32)])
        assert (x == 0).all()
        _, g = net.loss_grad([fv], [np.zeros((1, 4), np.float32)], [-zs], [np.zeros(1, np.float32)],
                             np.zeros(1, np.float32))
    o = {name: (at, shape) for name, at, shape, _ in lay.items}["Uv0"]
    dU = g[o[0]:o[0] + 64 * 64].reshape(64, 64)
    want = zs.astype(float).sum() * float(_float(h))          # 2^-16 of either product
    np.testing.assert_allclose(dU[0], want, rtol=2.0 ** -20)
    np.testing.assert_allclose(dU[1], -want, rtol=2.0 ** -20)
