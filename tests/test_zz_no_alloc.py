"""sps_kkt_noalloc: the KKT check that allocates no device memory.

Some callers cannot call cudaMalloc when they want a point checked: code that
runs inside another framework's memory pool or a fixed device-memory budget,
or a latency-critical loop where an allocation would synchronise the device.
For them the library offers one entry point whose scratch is a fixed array
inside the library; they pass the LP, the point and an output buffer, all in
device memory they already own.

The GPU test checks it, through the C ABI, twice in a row, against what the
existing entry point sps_solve reports for the same point (same tolerance form
as the other parity tests: 0.5 * tol absolute + 1e-3 relative, since sps_solve
evaluates with the FP32-rounded scaled matrix) and against the CPU oracle's FP64
evaluation (1e-9 relative plus 1e-12 absolute: both are FP64 sums of the same
products, in different orders).  Its K^T y is summed with integer digits, so
the two calls must agree bit for bit, on LPs whose columns hold 2 (transport),
about 10 (planted 200x500) and about 40 (planted 2000x4000) nonzeros; free
device memory must not change across calls.  This file is collected last.
"""

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
import sovereign_solver_gb300.workloads as wl
from sovereign_solver_gb300 import _native as N
from fixtures import load_problems
from oracle import kkt

TOL = 1e-5


def _case(name):
    if name == "planted":
        return wl.planted_lp(seed=11)[0]
    if name == "planted_dense":
        return wl.planted_lp(m=2000, n=4000, density=0.02, seed=3)[0]
    if name == "transport":
        return wl.transportation_lp(30, 60, seed=2)[0]
    return load_problems()["mixed_bounds"]


def _device_lp(torch, p):
    K = sp.vstack([sp.csr_matrix(p.A_ub, dtype=float), sp.csr_matrix(p.A_eq, dtype=float)], format="csr")
    rhs = np.concatenate([np.asarray(p.b_ub, float), np.asarray(p.b_eq, float)])
    dev = lambda a, dt: torch.tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")
    keep = [dev(K.indptr.astype(np.int32), torch.int32), dev(K.indices.astype(np.int32), torch.int32),
            dev(K.data, torch.float64), dev(p.c, torch.float64), dev(rhs, torch.float64),
            dev(p.lb, torch.float64), dev(p.ub, torch.float64)]
    lp = N.DeviceLP(p.n_vars, p.n_ineq, p.n_eq, *[t.data_ptr() for t in keep])
    return lp, keep


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["planted", "planted_dense", "transport", "mixed_bounds"])
def test_noalloc_kkt_matches_sps_solve(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = _case(name)
    with sps.PDHGEngine(p, tol=TOL, max_iters=200000) as eng:
        r = eng.solve_raw()
        x, y = eng.solution()
    assert r.status == 0
    lib = N.load()
    lp, keep = _device_lp(torch, p)
    xd = torch.tensor(x, dtype=torch.float64, device="cuda")
    yd = torch.tensor(y, dtype=torch.float64, device="cuda")
    out = torch.empty(6, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def call():
        out.fill_(float("nan"))
        rc = lib.sps_kkt_noalloc(C.byref(lp), xd.data_ptr(), yd.data_ptr(), out.data_ptr(), stream)
        assert rc == 0, lib.sps_last_error(None)
        torch.cuda.synchronize()
        return out.cpu().numpy().copy()

    call()      # the library's device module (and its static scratch) may load lazily on first use
    free0 = torch.cuda.mem_get_info()[0]
    calls = [call(), call()]
    assert torch.cuda.mem_get_info()[0] == free0, "free device memory changed across calls"
    engine = np.array([r.rel_kkt, r.rel_primal, r.rel_dual, r.rel_gap])
    box = kkt.box_rel_kkt(p, x, y)
    ref = np.array([box["err"], box["rp"], box["rd"], box["gap"], box["pobj"], box["dobj"]])
    for got in calls:
        assert np.all(np.isfinite(got))
        assert np.all(np.abs(got[:4] - engine) <= 0.5 * TOL + 1e-3 * np.abs(engine)), (got[:4], engine)
        np.testing.assert_allclose(got[:4], ref[:4], rtol=1e-9, atol=1e-12)
        np.testing.assert_allclose(got[4:], ref[4:], rtol=1e-9, atol=1e-12)
    assert np.array_equal(calls[0], calls[1]), calls


def test_noalloc_rejects_too_many_columns():
    """More columns than the fixed scratch holds: a clear error, no device work."""
    lib = N.load()
    lp = N.DeviceLP(300000, 0, 1, 8, 8, 8, 8, 8, 8, 8)
    rc = lib.sps_kkt_noalloc(C.byref(lp), 8, 8, 8, None)
    assert rc == -1
    assert b"262144" in lib.sps_last_error(None)


@pytest.mark.parametrize("missing", ["indptr", "indices", "values", "rhs", "c", "lb", "ub"])
def test_noalloc_rejects_null_arrays(missing):
    """A null device array where the LP needs one: a clear error before any device work
    (rows need indptr, indices, values and rhs even when they hold no nonzeros)."""
    lib = N.load()
    lp = N.DeviceLP(4, 1, 1, 8, 8, 8, 8, 8, 8, 8)
    setattr(lp, missing, None)
    rc = lib.sps_kkt_noalloc(C.byref(lp), 8, 8, 8, None)
    assert rc == -1
    assert b"null device array" in lib.sps_last_error(None)


@pytest.mark.gpu
@pytest.mark.parametrize("lengths,spread", [
    ([1, 7, 8, 9, 31, 32, 33, 255, 256, 257, 700, 0, 2], 0),     # around the lanes of a row and the long-row limit
    ([5] * 130, 0), ([0] * 40 + [1], 0), ([257] * 9, 0),         # (an LP without entries has null arrays: refused)
    ([12] * 70, 30),                                             # products over 60 decades: every digit, and below the last
])
def test_noalloc_kkt_row_schedules(lengths, spread):
    """Rows around the schedule's edges and products of very different sizes against FP64 sums
    (2 ** -50 of the sum of magnitudes: FP64 sums of at most 1500 terms in another order)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(5)
    m, n = len(lengths), 900
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lengths]).astype(np.int32)
    val = rng.standard_normal(idx.size) * 10.0 ** rng.uniform(-spread, spread, idx.size)
    A = sp.csr_matrix((val, idx, np.concatenate([[0], np.cumsum(lengths)])), shape=(m, n))
    k = m // 3
    p = sps.Problem(c=rng.standard_normal(n), A_ub=A[:k], b_ub=rng.standard_normal(k), A_eq=A[k:],
                    b_eq=rng.standard_normal(m - k), lb=np.zeros(n), ub=np.full(n, 3.0), integer_mask=np.zeros(n, bool))
    x, y = rng.random(n), rng.standard_normal(m)
    lib, (lp, keep) = N.load(), _device_lp(torch, p)
    xd, yd = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (x, y))
    outs = []
    for _ in range(2):
        out = torch.full((6,), float("nan"), dtype=torch.float64, device="cuda")
        assert lib.sps_kkt_noalloc(C.byref(lp), xd.data_ptr(), yd.data_ptr(), out.data_ptr(), None) == 0
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    rhs = np.concatenate([p.b_ub, p.b_eq])
    res = A @ x - rhs
    res[:k] = np.maximum(res[:k], 0)
    rc = p.c - A.T @ y
    po, do = p.c @ x, rhs @ y + 3.0 * np.minimum(rc, 0).sum()
    eps = 2.0 ** -50
    assert abs(outs[0][1] - np.linalg.norm(res) / (1 + np.linalg.norm(rhs))) <= eps * (1 + np.linalg.norm(abs(A) @ x))
    assert abs(outs[0][4] - po) <= eps * (abs(p.c) @ x)
    assert abs(outs[0][5] - do) <= eps * (abs(rhs) @ abs(y) + 3.0 * (abs(p.c) + abs(A).T @ abs(y)).sum())
