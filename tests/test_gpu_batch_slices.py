"""Batched solve: the slice layout of the passes at the sizes where it can go wrong.

Chunk edges (a warp takes 32 / lanes rows at once), one row or column, empty rows
and columns, an instance without entries, a row so long that its side stays on
the CSR, vectors past the staging buffer, and a team.  Every instance is checked
by the CPU oracle in FP64, with the tolerances of the batch tests.
"""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
import sovereign_solver_gb300.workloads as wl
from oracle import kkt

pytestmark = pytest.mark.gpu

TOL = 1e-4


def _box(A, seed, name):
    """min c x over A x <= b, 0 <= x <= 1, with b that x = 1/4 meets."""
    rng = np.random.default_rng(seed)
    A = sp.csr_matrix(A)
    m, n = A.shape
    return sps.Problem(c=rng.standard_normal(n), A_ub=A, b_ub=A @ np.full(n, 0.25) + rng.uniform(0.1, 1.0, m),
                       A_eq=sp.csr_matrix((0, n)), b_eq=np.zeros(0), lb=np.zeros(n), ub=np.ones(n),
                       integer_mask=np.zeros(n, dtype=bool), name=name)


def _shapes():
    rng = np.random.default_rng(7)
    dense = lambda m, n: rng.uniform(0.5, 1.5, (m, n))                                     # noqa: E731
    out = [_box(dense(m, n), m * 100 + n, f"dense_{m}x{n}")
           for m, n in ((1, 1), (1, 70), (70, 1), (31, 33), (32, 32), (33, 31), (8, 257), (257, 8))]
    sparse = sp.random(90, 130, density=0.05, random_state=3, format="lil")
    sparse[7, :] = 0.0
    sparse[:, 11] = 0.0
    sparse[89, :] = 0.0
    out.append(_box(sparse, 1, "empty_row_and_column"))
    out.append(_box(sp.csr_matrix((5, 9)), 2, "no_entries"))
    long_row = sp.lil_matrix((300, 2000))
    for i in range(300):
        long_row[i, rng.integers(0, 2000, 2)] = 1.0
    long_row[150, :] = rng.uniform(0.5, 1.5, 2000)
    out.append(_box(long_row, 4, "one_long_row"))
    wide = sp.random(40, 9000, density=0.02, random_state=5, format="csr")
    out.append(_box(wide, 5, "past_the_staging_buffer"))
    return out


def _check(p, r):
    assert r.status == "optimal", (p.name, r)
    box = kkt.box_rel_kkt(p, r.x, r.y)
    assert box["err"] < 1.5 * TOL, (p.name, box)


@pytest.mark.parametrize("group", [1, 2, 8, 32])
def test_slices_at_the_edges(group):
    probs = _shapes()
    with sps.PDHGBatch(probs, tol=TOL, max_iters=200000, batch_group=group) as b:
        res = b.solve()
    for p, r in zip(probs, res):
        _check(p, r)


def test_slices_of_a_team():
    probs = [wl.batch_planted_lp(k, m_range=(60, 300))[0] for k in range(12)]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=200000, batch_team=4, batch_team_nnz=2000) as b:
        res = b.solve()
        assert b.stats.team == 4
    for p, r in zip(probs, res):
        _check(p, r)


@pytest.mark.parametrize("kind", ["planted", "two_entry_columns", "mixed"])
def test_more_instances_than_sms(kind):
    """Two blocks on an SM (the batches above run one): sliced, on the CSR, and some of each."""
    planted = [wl.batch_planted_lp(k, m_range=(40, 90))[0] for k in range(200)]
    short = [wl.transportation_lp(5 + k % 7, 9 + k % 5, seed=k)[0] for k in range(200)]
    probs = {"planted": planted, "two_entry_columns": short, "mixed": planted + short}[kind]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=200000) as b:
        res = b.solve()
        assert b.stats.blocks > 152
    for p, r in zip(probs, res):
        _check(p, r)
