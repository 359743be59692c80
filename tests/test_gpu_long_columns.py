"""LPs with columns of over 512 nonzeros (SEGMENT columns), in both error forms: the PDLP
form's check leaves 18 partials per such column.  Points re-checked by the CPU oracle in
the same form; the same bits from a second solve."""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from oracle import kkt

pytestmark = pytest.mark.gpu


def _narrow(m, n, seed):
    """m rows on n columns, every entry there: columns of m nonzeros."""
    rng = np.random.default_rng(seed)
    A = sp.csr_matrix(rng.uniform(0.2, 1.0, (m, n)) * rng.choice([-1.0, 1.0], (m, n)))
    x, k = rng.random(n), m // 3
    return sps.Problem(c=rng.standard_normal(n), A_ub=A[:k], b_ub=A[:k] @ x + rng.uniform(0.1, 1.0, k), A_eq=A[k:],
                       b_eq=A[k:] @ x, lb=np.zeros(n), ub=np.ones(n), integer_mask=np.zeros(n, bool)), x


@pytest.mark.parametrize("form", ["pdlp", "lagrangian"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("m,n", [(513, 1), (700, 2), (1454, 4), (600, 17)])
def test_long_columns(m, n, precision, form):
    p, x = _narrow(m, n, m + n)
    tol = 1e-4
    with sps.PDHGEngine(p, tol=tol, precision=precision, kkt_form=form, max_iters=20000) as e:
        a, b = e.solve(), e.solve()
    assert a.status == "optimal" and np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    assert kkt.box_rel_kkt(p, a.x, a.y, form=form)["err"] < 1.5 * tol
    if n <= m - m // 3:
        assert np.abs(a.x - x).max() < 0.05                    # the '=' rows alone fix x


@pytest.mark.parametrize("form", ["pdlp", "lagrangian"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("m,n", [(700, 2), (600, 17), (2000, 40)])
def test_rejected_attempts(m, n, precision, form):
    """From an optimal point the first attempts are rejected; their movement is the candidate's own
    (the long columns' slots hold another kernel's sums then)."""
    p, _ = _narrow(m, n, m + n)
    tol = 1e-4
    with sps.PDHGEngine(p, tol=tol, precision=precision, kkt_form=form, max_iters=20000) as e:
        a = e.solve()
        e.warm_start(a.x, a.y)
        b = e.solve()
    assert a.status == "optimal" and b.status == "optimal" and b.iterations <= a.iterations
    assert b.stats["step_size"] > 0 and b.stats["accepted_steps"] < b.iterations
    assert kkt.box_rel_kkt(p, b.x, b.y, form=form)["err"] < 1.5 * tol
