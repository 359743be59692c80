"""The two layouts of a batch's matrices give the same bits: every case solves with the
slices, gives them back (which says whether there were any) and solves on the CSR."""

import numpy as np
import pytest

import sovereign_solver_gb300 as sps
import sovereign_solver_gb300.workloads as wl
from test_gpu_batch_slices import TOL, _shapes

pytestmark = pytest.mark.gpu


def _both(b, slices=True):
    got = [b.solve()]
    assert b.lib.sps_batch_release_slices(b.h) == (1 if slices else 0)
    assert b.lib.sps_batch_release_slices(b.h) == 0
    got.append(b.solve())
    for r, q in zip(*got):
        assert (r.status, r.iterations, r.rel_kkt, r.objective) == (q.status, q.iterations, q.rel_kkt, q.objective)
        assert np.array_equal(r.x, q.x) and np.array_equal(r.y, q.y)
    return got[0]


@pytest.mark.parametrize("group", [1, 2, 8, 32])
@pytest.mark.parametrize("graph_mode", [0, 2])
def test_edges(group, graph_mode):
    with sps.PDHGBatch(_shapes(), tol=TOL, max_iters=20000, batch_group=group, escalate="off",
                       graph_mode=graph_mode) as b:
        _both(b)


@pytest.mark.parametrize("team", [2, 4, 8])
def test_teams(team):
    probs = [wl.batch_planted_lp(k, m_range=(60, 300))[0] for k in range(12)]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=20000, batch_team=team, batch_team_nnz=2000, escalate="off") as b:
        _both(b)
        assert b.stats.team == team


@pytest.mark.parametrize("kind", ["planted", "two_entry_columns", "mixed"])
def test_more_instances_than_sms(kind):
    planted = [wl.batch_planted_lp(k, m_range=(40, 90))[0] for k in range(200)]
    short = [wl.transportation_lp(5 + k % 7, 9 + k % 5, seed=k)[0] for k in range(200)]
    probs = {"planted": planted, "two_entry_columns": short, "mixed": planted + short}[kind]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=2000, escalate="off") as b:
        _both(b, slices=kind != "two_entry_columns")


def test_warm_starts():
    """The cold starts' errors are kept by the first solve, and the warm points are judged by them in both."""
    probs = [wl.batch_planted_lp(k, m_range=(60, 200))[0] for k in range(24)]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=20000, escalate="off") as b:
        cold = b.solve()
        b.set_warm_starts([(r.x, r.y, None) for r in cold])
        warm = _both(b)
        assert sum(r.iterations for r in warm) < sum(r.iterations for r in cold) / 2


def test_grid_is_what_is_resident():
    """A launch has no blocks that wait for others to end (they would count as idle for the
    hand-off): two on an SM with slices, four on the CSR; whole clusters with teams."""
    probs = [wl.batch_planted_lp(k, m_range=(40, 60))[0] for k in range(640)]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=200, escalate="off") as b:
        b.solve_raw()
        sliced = b.stats.blocks
        assert b.lib.sps_batch_release_slices(b.h) == 1
        b.solve_raw()
        assert (sliced, b.stats.blocks) == (2 * 152, 4 * 152)
    with sps.PDHGBatch(probs[:60], tol=TOL, max_iters=200, escalate="off", batch_team=8, batch_team_nnz=100) as b:
        b.solve_raw()
        assert b.stats.team == 8 and b.stats.blocks % 8 == 0 and b.stats.blocks <= 2 * 152
        assert b.lib.sps_batch_release_slices(b.h) == 1
        b.solve_raw()
        assert b.stats.blocks == 480


def test_teams_are_resident_at_once():
    """19 clusters of 8 blocks do not all fit one block per SM: they take the form of two."""
    probs = [wl.batch_planted_lp(k, m_range=(60, 300))[0] for k in range(19)]
    with sps.PDHGBatch(probs, tol=TOL, max_iters=20000, batch_team=8, batch_team_nnz=500, escalate="off") as b:
        _both(b)
        assert (b.stats.team, b.stats.blocks) == (8, 152)


def test_teams_do_not_wait_for_one_another():
    """16 teams of 8 blocks take 1.3 times as long as 12 (1.9 times where two teams waited)."""
    probs = [wl.batch_planted_lp(k, m_range=(1500, 1500), n_ratio=(2.0, 2.0))[0] for k in range(16)]

    def best(count):
        with sps.PDHGBatch(probs[:count], tol=1e-12, max_iters=640, escalate="off") as b:
            ms = [b.solve_raw().solve_ms for _ in range(6)]
            assert b.stats.team == 8
            return min(ms[1:])
    assert best(16) < 1.6 * best(12)


def test_every_large_instance_gets_its_team():
    """Instances of many columns but few nonzeros lie among the large ones in the order of work; a
    cluster that met one broke up, and the large ones after it were solved by a team or by one
    block as it happened.  Each has the bits that it has in a batch of large ones alone."""
    import scipy.sparse as sp

    def box(m, n, per_row, seed):
        rng = np.random.default_rng(seed)
        A = sp.csr_matrix((rng.standard_normal(m * per_row),
                           np.concatenate([rng.choice(n, per_row, replace=False) for _ in range(m)]),
                           np.arange(0, m * per_row + 1, per_row)), shape=(m, n))
        return sps.Problem(c=rng.standard_normal(n), A_ub=A, b_ub=A @ np.full(n, 0.25) + rng.uniform(0.1, 1.0, m),
                           A_eq=sp.csr_matrix((0, n)), b_eq=np.zeros(0), lb=np.zeros(n), ub=np.ones(n),
                           integer_mask=np.zeros(n, bool))
    first = [box(300, 600, 20, k) for k in range(40)]                      # work 6900, 6000 nonzeros
    sparse = [box(40, 4000, 10, 100 + k) for k in range(60)]               # work 4440, 400 nonzeros
    last = [box(60, 150, 20, 200 + k) for k in range(120)]                 # work 1410, 1200 nonzeros
    opts = dict(tol=1e-9, max_iters=640, escalate="off", batch_group=4, batch_team=8, batch_team_nnz=1000)
    with sps.PDHGBatch(first + last, **opts) as b:
        alone = b.solve()
        lanes = b.stats.lanes_per_row
    with sps.PDHGBatch(first + sparse + last, **opts) as b:
        mixed = b.solve()
        assert b.stats.team == 8
        if b.stats.lanes_per_row != lanes:
            pytest.skip("the two batches timed another schedule")
    for r, q in zip(alone, mixed[:40] + mixed[100:]):
        assert np.array_equal(r.x, q.x) and np.array_equal(r.y, q.y) and r.iterations == q.iterations
