"""GPU parity at the edges of the launch rules: mesh classes around the bounds between the
resident solvers (up to three cells per thread of a CTA of at most 512), the general solvers
and the thread-block clusters (above 1536 cells), and linear systems around the bounds of
their row slices, CTA-local levels and cluster sizes.

Tolerances: the flow fields after a few outer iterations differ from the restatement by the
order of sums (1e-9 of the field's scale, as in the other trajectory tests); a linear solution
from its direct one by the requested residual 1e-10 times the condition number of the
system (below 100 for the diagonally dominant ones: 1e-8; 1e-7 for the Poisson systems).
"""
import numpy as np
import pytest

import cases
import rans_uq_b200.linear as lin
import rans_uq_b200.workloads as wl
from oracle import checker as ck

pytestmark = pytest.mark.gpu
RTOL = 1e-9
ITERS = 6


def check_fields(rq, checker, case, solver="AMG", block=0):
    want = checker.solve(case, "oracle")
    batch = cases.product_batch(rq, case, pressure_solver=solver, block_threads=block)
    res, fields, _ = batch.evaluate_fields([[case.coeffs[9], case.coeffs[8]]])
    assert res.rows[0].result.status.name == want.status
    assert res.rows[0].result.simple_iters == want.iterations
    u = max(np.max(np.abs(want.field("Ux"))), 1e-300)
    for name in ("Ux", "k", "omega", "nuT", "F1"):
        i = ck.FIELD_NAMES.index(name)
        scale = max(np.max(np.abs(want.fields[i])), 1e-300)
        assert np.max(np.abs(fields[0, i] - want.fields[i])) / scale < RTOL, name
    assert np.max(np.abs(fields[0, 1] - want.field("Uy"))) / u < RTOL
    pscale = max(np.max(np.abs(want.field("p"))), 1.0)
    assert np.max(np.abs(fields[0, 3] - want.field("p"))) / pscale < RTOL


@pytest.mark.parametrize("nx,ny", [(3, 2), (3, 3), (3, 32), (4, 25), (5, 103), (3, 341), (3, 512),
                                   (3, 513)])
def test_channel_sizes(rq, checker, nx, ny):
    check_fields(rq, checker, cases.small_channel(nx=nx, ny=ny, max_iter=ITERS))


@pytest.mark.parametrize("nx,ny", [(45, 28), (48, 32), (49, 32), (64, 40)])
def test_bump_sizes(rq, checker, nx, ny):
    check_fields(rq, checker, cases.bump_case(nx, ny, max_iter=ITERS))


@pytest.mark.parametrize("solver,ps", [("AMG", ck.P_AMG), ("PCG", ck.P_PCG)])
@pytest.mark.parametrize("block", [64, 128, 256, 512, 768, 1024])
def test_block_sizes(rq, checker, block, solver, ps):
    check_fields(rq, checker, cases.small_channel(ny=64, max_iter=ITERS, pressure_solver=ps), solver,
                 block)


def test_cluster_rows_independent_of_batch(rq):
    case = cases.bump_case(60, 36, max_iter=ITERS)
    batch = cases.product_batch(rq, case)
    theta = np.array([[0.29, 0.085], [0.31, 0.09], [0.33, 0.095]])
    alone = [batch.evaluate(theta[i:i + 1]).predictions[0] for i in range(3)]
    together = batch.evaluate(np.concatenate([theta] * 20)).predictions
    for i, row in enumerate(together):
        np.testing.assert_array_equal(row, alone[i % 3])


def test_cluster_without_allocation_equals_batch(rq):
    from test_zz_no_alloc import _noalloc_two_calls

    _noalloc_two_calls(rq, cases.bump_case(60, 36, max_iter=ITERS),
                       np.array([[0.31, 0.09], [0.33, 0.092]]))


def test_mixed_cluster_equals_mixed_single_cta(rq):
    """The FP32 inner solves round differently (1e-7 per correction): 1e-5 after 6 iterations."""
    case = cases.bump_case(60, 36, max_iter=ITERS)
    theta = [[case.coeffs[9], case.coeffs[8]]]
    a = cases.product_batch(rq, case, precision="mixed").evaluate(theta).predictions
    b = cases.product_batch(rq, case, precision="mixed", block_threads=512).evaluate(theta).predictions
    assert np.max(np.abs(a - b)) / np.max(np.abs(b)) < 1e-5


# ---------------------------------------------------------------- linear systems
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [5, 6, 33, 45, 46, 64])
def test_poisson_around_slices_and_clusters(n, precision):
    s = wl.poisson_system(n, 40 + n)
    dense = np.diag(s.diag)
    dense[s.own, s.nbr] = s.upper
    dense[s.nbr, s.own] = s.lower
    (r,), (x,) = lin.solve_batch([s], kind="AMG", precision=precision, max_iter=500, tol=1e-10)
    want = np.linalg.solve(dense, s.source)
    assert r.converged
    assert np.linalg.norm(x - want) / np.linalg.norm(want) < 1e-7


@pytest.mark.parametrize("kind", ["PCG", "BiCGSTAB"])
@pytest.mark.parametrize("n", [31, 300, 5000])
def test_one_long_row(n, kind):
    """A star: one row of n entries (plain CSR rows), the others of two."""
    own, nbr = np.zeros(n - 1, np.int32), np.arange(1, n, dtype=np.int32)
    c = np.full(n - 1, -0.5 / n)
    rng = np.random.default_rng(n)
    b = rng.standard_normal(n)
    s = lin.LinearSystem.from_arrays(np.ones(n), c, c, b, own, nbr)
    (r,), (x,) = lin.solve_batch([s], kind=kind, max_iter=200, tol=1e-10)
    # x_0 = (b_0 - c sum b_i) / (1 - (n - 1) c^2), x_i = b_i - c x_0
    x0 = (b[0] - c[0] * b[1:].sum()) / (1 - (n - 1) * c[0] ** 2)
    want = np.concatenate([[x0], b[1:] - c[0] * x0])
    assert r.converged
    assert np.linalg.norm(x - want) / np.linalg.norm(want) < 1e-8


def test_uneven_batch_equals_single_solves():
    sizes = [9, 64, 33, 100, 46]
    systems = [wl.poisson_system(n, 60 + n) for n in sizes]
    results, xs = lin.solve_batch(systems, kind="AMG", max_iter=500, tol=1e-10)
    for s, r, x in zip(systems, results, xs):
        (r1,), (x1,) = lin.solve_batch([s], kind="AMG", max_iter=500, tol=1e-10)
        assert r1.iterations == r.iterations
        np.testing.assert_array_equal(x1, x)
