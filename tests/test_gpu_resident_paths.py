"""Which LPs run a window in one resident launch, told by the launches they report, in both
modes; the bits at the sizes that only the reference mode's smaller state lets in; and
that the transportation LPs of test_gpu_resident do reject attempts."""

import numpy as np
import pytest

import sovereign_solver_gb300 as sps
import sovereign_solver_gb300.workloads as wl
from test_gpu_resident import LPS, WAVE

pytestmark = pytest.mark.gpu


def _solve(p, mode, precision, **kw):
    its = 5 * (64 if mode == "adaptive" else 50) + 23
    with sps.PDHGEngine(p, mode=mode, precision=precision, tol=1e-13, max_iters=its, escalate="off", **kw) as e:
        e.solve()
        return e.solve()


def _resident(launched, other):
    return other.stats["kernel_launches"] < launched.stats["kernel_launches"] / 4


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("name", list(LPS))
def test_path_in_reference_mode(name, precision):
    make, in32, in64 = LPS[name]
    p = make()
    want = in32 if precision == "fp32" else in64 and name != "2003x5009"       # upper bounds are rows here: too large
    a, b = (_solve(p, "reference", precision, **kw) for kw in ({"max_blocks": WAVE}, {}))
    assert a.iterations == b.iterations
    if a.iterations >= 100:                # two windows or more
        assert _resident(a, b) == want


@pytest.mark.parametrize("make,precision,resident", [
    (lambda: wl.transportation_lp(80, 160, seed=1)[0], "fp64", True),
    (lambda: wl.transportation_lp(90, 180, seed=1)[0], "fp64", True),
    (lambda: wl.transportation_lp(100, 200, seed=1)[0], "fp64", False),        # 320 column tasks for 256 warps
    (lambda: wl.transportation_lp(120, 240, seed=1)[0], "fp32", True),
    (lambda: wl.planted_lp(3000, 7500, 0.003, seed=1)[0], "fp32", True),
    (lambda: wl.planted_lp(1500, 3700, 0.007, seed=1)[0], "fp64", True),
])
def test_reference_mode_has_its_own_capacity(make, precision, resident):
    p = make()
    a, b = (_solve(p, "reference", precision, **kw) for kw in ({"max_blocks": WAVE}, {}))
    assert _resident(a, b) == resident
    assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    assert (a.status, a.iterations, a.objective, a.rel_kkt) == (b.status, b.iterations, b.objective, b.rel_kkt)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("name", ["transport_20x31", "transport_37x53"])
def test_attempts_are_rejected(name, precision):
    for kw in ({"max_blocks": WAVE}, {}):
        r = _solve(LPS[name][0](), "adaptive", precision, **kw)
        assert r.stats["accepted_steps"] < r.iterations
