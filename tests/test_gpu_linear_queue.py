"""How many CTAs a system of a batch takes depends on the batch; its sums are formed in the same
slices whatever that number, so its solution equals that of the system alone bit for bit."""
import numpy as np
import pytest

import rans_uq_b200.linear as lin
import rans_uq_b200.workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision", [("AMG", "fp64"), ("AMG", "mixed"), ("PCG", "fp64"),
                                            ("PCG", "mixed"), ("BiCGSTAB", "fp64")])
@pytest.mark.parametrize("n", [45, 46, 64, 130])  # 1, 2, 4 and 16 slices
def test_solutions_do_not_depend_on_the_number_of_systems(n, kind, precision):
    systems = [wl.poisson_system(n, 80 + k) for k in range(3)]
    alone = [lin.solve_batch([s], kind=kind, precision=precision, max_iter=2000, tol=1e-8)
             for s in systems]
    for count in (4, 12, 40, 80, 160):
        results, xs = lin.solve_batch([systems[k % 3] for k in range(count)], kind=kind,
                                      precision=precision, max_iter=2000, tol=1e-8)
        for k, (r, x) in enumerate(zip(results, xs)):
            (r1,), (x1,) = alone[k % 3]
            assert r.converged and r.iterations == r1.iterations
            np.testing.assert_array_equal(x, x1)


def test_mixed_sizes():
    sizes = [300] * 4 + [130] * 30 + [64] * 60 + [20] * 60
    systems = [wl.poisson_system(n, 90 + k % 2) for k, n in enumerate(sizes)]
    results, xs = lin.solve_batch(systems, kind="AMG", max_iter=500, tol=1e-10)
    for k in (0, 3, 4, 33, 34, 93, 94, 153):
        (r1,), (x1,) = lin.solve_batch([systems[k]], kind="AMG", max_iter=500, tol=1e-10)
        assert results[k].converged and results[k].iterations == r1.iterations
        np.testing.assert_array_equal(xs[k], x1)


def test_solutions_of_small_and_large_systems_in_any_order():
    """Runs of small solutions are read back together, those of 12288 rows and more alone."""
    sizes = [20, 111, 8, 9, 110, 10, 112, 113, 5, 40]
    systems = [wl.poisson_system(n, 70 + k) for k, n in enumerate(sizes)]
    batch = lin.LinearBatch(systems, kind="AMG")
    _, zero = batch.solve(500, 1e-10)
    _, start = batch.solve(500, 1e-10, xs=[np.zeros(s.n_cells) for s in systems])
    for s, x, y in zip(systems, zero, start):
        (_,), (x1,) = lin.solve_batch([s], kind="AMG", max_iter=500, tol=1e-10)
        np.testing.assert_array_equal(x, x1)
        np.testing.assert_array_equal(y, x1)
