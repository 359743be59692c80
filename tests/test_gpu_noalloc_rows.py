"""sps_kkt_noalloc around the edges of its row schedules: 32, 16 and 8 lanes a row (by the
number of rows), rows at and above the length that a whole warp takes, alone and in
clumps; and its time on few long rows and on wide LPs of few rows."""

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import sovereign_solver_gb300 as sps
from sovereign_solver_gb300 import _native as N
from test_zz_no_alloc import _device_lp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lp(m, n, lengths, seed=5):
    rng = np.random.default_rng(seed)
    ptr = np.concatenate([[0], np.cumsum(lengths)])
    step = np.repeat(np.maximum(n // np.maximum(lengths, 1), 1), lengths)
    idx = ((np.arange(ptr[-1]) - np.repeat(ptr[:-1], lengths)) * step).astype(np.int32)      # distinct, rising
    A = sp.csr_matrix((rng.standard_normal(ptr[-1]), idx, ptr), shape=(m, n))
    k = m // 3
    p = sps.Problem(c=rng.standard_normal(n), A_ub=A[:k], b_ub=rng.standard_normal(k), A_eq=A[k:],
                    b_eq=rng.standard_normal(m - k), lb=np.zeros(n), ub=np.full(n, 3.0), integer_mask=np.zeros(n, bool))
    return p, A, rng.random(n), rng.standard_normal(m)


class _Call:
    def __init__(self, p, x, y):
        self.lib = N.load()
        self.lp, self.keep = _device_lp(torch, p)
        self.x, self.y = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (x, y))
        self.out = torch.full((6,), float("nan"), dtype=torch.float64, device="cuda")

    def __call__(self):
        assert self.lib.sps_kkt_noalloc(C.byref(self.lp), self.x.data_ptr(), self.y.data_ptr(), self.out.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream) == 0
        return self.out

    def best_ms(self):
        ts = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            self()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts[3:])


@pytest.mark.parametrize("m", [1, 9, 1216, 1217, 2432, 2433, 33000])
def test_lanes_and_long_rows(m):
    """2^-44 of the sum of magnitudes: no sum here has a chain of more than 500 FP64 additions."""
    lengths = np.full(m, 3)
    lengths[m // 2:m // 2 + 70] = 300                       # a clump of long rows
    lengths[:4] = (255, 256, 257, 0)[:m] if m < 4 else (255, 256, 257, 0)
    lengths[-1] = 700
    p, A, x, y = _lp(m, 900, lengths)
    call = _Call(p, x, y)
    out, again = call().cpu().numpy().copy(), call().cpu().numpy()
    assert np.array_equal(out, again)
    rhs = np.concatenate([p.b_ub, p.b_eq])
    res = A @ x - rhs
    res[:m // 3] = np.maximum(res[:m // 3], 0)
    rc = p.c - A.T @ y
    eps = 2.0 ** -44
    assert abs(out[1] - np.linalg.norm(res) / (1 + np.linalg.norm(rhs))) <= eps * (1 + np.linalg.norm(abs(A) @ x))
    assert abs(out[4] - p.c @ x) <= eps * (abs(p.c) @ x)
    assert abs(out[5] - (rhs @ y + 3.0 * np.minimum(rc, 0).sum())) <= \
        eps * (abs(rhs) @ abs(y) + 3.0 * (abs(p.c) + abs(A).T @ abs(y)).sum())


def test_long_rows_run_side_by_side():
    """Four rows of 20 000 nonzeros take as long as one (3.7 times where one warp took the four)."""
    ms = [_Call(*(v for k, v in enumerate(_lp(m, 80_000, np.full(m, 20_000))) if k != 1)).best_ms() for m in (1, 4)]
    assert ms[1] < 2 * ms[0]


def test_few_rows_clear_all_columns_together():
    """262 144 columns under 10 short rows against 40 000 rows on as many columns: less work,
    less time (six times as long where one block cleared the columns' sums)."""
    ms = [_Call(*(v for k, v in enumerate(_lp(m, 262_144, np.full(m, 20))) if k != 1)).best_ms() for m in (10, 40_000)]
    assert ms[0] < ms[1]
