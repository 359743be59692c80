"""The resident window kernel (one launch per window of attempts, for LPs that one
thread-block cluster holds) against the launched passes: the same bits.

``max_blocks`` at one resident wave (760 blocks, the default plan) keeps the
launched passes, so both runs share the plan and differ only in the kernel.
"""

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
import sovereign_solver_gb300.workloads as wl
from sovereign_solver_gb300.problem import Problem

WAVE = 760


def _bounds(p, seed):
    """p with mixed finite and infinite bounds and every row kind."""
    rng = np.random.default_rng(seed)
    n = p.n_vars
    lb = np.where(rng.random(n) < 0.3, -np.inf, -rng.random(n))
    ub = np.where(rng.random(n) < 0.3, np.inf, 1.0 + rng.random(n))
    k = p.A_eq.shape[0] // 2
    return Problem(c=p.c, A_ub=p.A_eq[:k], b_ub=p.b_eq[:k], A_eq=p.A_eq[k:], b_eq=p.b_eq[k:], lb=lb, ub=ub,
                   integer_mask=p.integer_mask)


def _dense_row(m, n, seed):
    """A row of n nonzeros above m short ones: longer than 512, it keeps the launched passes."""
    rng = np.random.default_rng(seed)
    A = sp.vstack([sp.csr_matrix(rng.random((1, n)) + 0.1), sp.random(m, n, 0.05, random_state=seed)]).tocsr()
    x = rng.random(n)
    return Problem(c=rng.random(n), A_ub=A, b_ub=A @ x, A_eq=sp.csr_matrix((0, n)), b_eq=np.zeros(0),
                   lb=np.zeros(n), ub=np.ones(n), integer_mask=np.zeros(n, bool))


# name: (problem, resident in FP32, in FP64).  Clusters of 1, 2, 4, 8 and 16 blocks; SLICED, WARP and
# SLAB rows (of one and of several units); slices with remainders; sizes below one warp.
LPS = {
    "1x1": (lambda: wl.planted_lp(1, 1, 1.0, seed=3)[0], True, True),
    "3x40": (lambda: wl.planted_lp(3, 40, 0.9, seed=3)[0], True, True),
    "33x65": (lambda: wl.planted_lp(33, 65, 0.2, seed=5)[0], True, True),
    "64x128_bounds": (lambda: _bounds(wl.planted_lp(64, 128, 0.2, seed=7)[0], 1), True, True),
    "200x500": (lambda: wl.planted_lp(seed=2)[0], True, True),
    "60x400_warp_rows": (lambda: wl.planted_lp(60, 400, 0.6, seed=8)[0], True, True),
    "transport_20x31": (lambda: wl.transportation_lp(20, 31, seed=1)[0], True, True),
    "transport_37x53": (lambda: wl.transportation_lp(37, 53, seed=1)[0], True, True),
    "1000x2500": (lambda: wl.planted_lp(1000, 2500, 0.01, seed=1)[0], True, True),
    "2003x5009": (lambda: wl.planted_lp(2003, 5009, 0.005, seed=1)[0], True, True),
    "transport_100x200": (lambda: wl.transportation_lp(100, 200, seed=1)[0], True, False),
    "dense_row_30x600": (lambda: _dense_row(30, 600, 1), False, False),
    "6000x15000": (lambda: wl.planted_lp(6000, 15000, 0.0015, seed=1)[0], False, False),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(LPS))
@pytest.mark.parametrize("mode,precision", [("adaptive", "fp32"), ("adaptive", "fp64"),
                                            ("reference", "fp32"), ("reference", "fp64")])
def test_resident_equals_launched_passes(name, mode, precision):
    make, in32, in64 = LPS[name]
    p = make()
    # ends inside a window, after restarts; a rejected attempt or more on the transportation LPs
    its = 5 * (64 if mode == "adaptive" else 50) + 23
    got = []
    for extra in ({"max_blocks": WAVE}, {}):
        with sps.PDHGEngine(p, mode=mode, precision=precision, tol=1e-13, max_iters=its, escalate="off", **extra) as e:
            e.solve()
            r = e.solve()                       # a second solve from the engine's own buffers
        got.append(r)
    a, b = got
    assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    assert (a.status, a.iterations, a.objective, a.rel_kkt) == (b.status, b.iterations, b.objective, b.rel_kkt)
    for k in ("restarts", "accepted_steps", "primal_weight", "step_size", "returned_average"):
        assert a.stats[k] == b.stats[k], k
    if a.iterations == its and mode == "adaptive":        # which path ran, where the plan does not depend on mode
        assert (b.stats["kernel_launches"] < a.stats["kernel_launches"] / 4) == (in32 if precision == "fp32" else in64)


@pytest.mark.gpu
@pytest.mark.parametrize("graph_mode", [0, 1, 2])
def test_resident_solve_to_tolerance(graph_mode):
    """To the tolerance, through a stall and its FP64 continuation, in every graph mode."""
    p = wl.planted_lp(60, 150, 0.15, seed=4)[0]
    got = []
    for extra in ({"max_blocks": WAVE}, {}):
        with sps.PDHGEngine(p, tol=1e-8, max_iters=20000, graph_mode=graph_mode, **extra) as e:
            got.append(e.solve())
    a, b = got
    assert a.status == "optimal" and np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    assert (a.iterations, a.rel_kkt, a.stats["escalated"]) == (b.iterations, b.rel_kkt, b.stats["escalated"])
