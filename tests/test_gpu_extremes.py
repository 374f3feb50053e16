"""Coefficients whose products leave the normal range: rq_solve takes any positive beta*, and
the closure divides by beta* omega y. The quotients that overflow are bounded by the closure's
own minima, so a subnormal divisor gives the solve of a tiny normal one (equal up to terms of
the order of beta* itself: 1e-12 of each field's scale)."""
import ctypes as C

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [24, 513])  # resident solvers, a cluster
def test_subnormal_beta_star(rq, ny):
    import rans_uq_b200._native as N

    case = cases.small_channel(ny=ny, max_iter=30, turb_start=2, nut_floor_iters=4)
    batch = cases.product_batch(rq, case)
    n = batch._problem.n_cells

    def solve(beta_star):
        coeffs = np.array(case.coeffs, dtype=float)
        coeffs[8] = beta_star
        row, pred, f = N.RowOut(), np.zeros(len(case.obs_x)), np.zeros((11, n))
        N.call("rq_solve", batch._problem.handle, N.dptr(coeffs), C.byref(row), N.dptr(pred),
               N.dptr(f), None, C.c_int32(0))
        return row, f

    want_row, want = solve(1e-280)
    row, got = solve(1e-310)
    assert row.status == want_row.status == int(rq.EvaluationStatus.Unconverged)
    assert row.iterations == want_row.iterations
    for w, g in zip(want, got):
        assert np.all(np.isfinite(w)) and np.max(np.abs(w)) >= 0
        assert np.max(np.abs(g - w)) <= 1e-12 * max(np.max(np.abs(w)), 1e-200)
