"""Solves on thread-block clusters (classes above 1536 cells).

How many CTAs a solve takes depends on the number of draws; its sums are formed in the same
slices whatever that number, so rows equal those of a draw alone bit for bit.

The CTAs of a cluster share the level vectors in global memory and run the small AMG levels
whole, each for itself. A CTA that reads a vector which another has overwritten shows as a row
that differs between equal draws or between launches, or as fields away from the
restatement's (1e-9 of the scale after a few outer iterations: the order of sums).
"""
import numpy as np
import pytest

import cases
from test_gpu_dispatch import check_fields

pytestmark = pytest.mark.gpu
ITERS = 6


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(60, 36), (100, 50)])  # first level in every CTA: 1 and 2
def test_equal_draws_and_launches_give_equal_rows(rq, nx, ny, precision):
    case = cases.bump_case(nx, ny, max_iter=20)
    batch = cases.product_batch(rq, case, precision=precision)
    theta = np.repeat([[0.31, 0.09]], 40, axis=0)
    first, fields, _ = batch.evaluate_fields(theta)
    again, fields2, _ = batch.evaluate_fields(theta)
    for f in list(fields) + list(fields2):
        np.testing.assert_array_equal(f, fields[0])
    for p in np.concatenate([first.predictions, again.predictions]):
        np.testing.assert_array_equal(p, first.predictions[0])


def test_inadmissible_draws_between_admissible_ones(rq):
    """An out-of-bounds draw passes no cluster barrier of its solve; the clusters' job queue
    stays in step over single ones, runs of them, and a batch of nothing else."""
    case = cases.bump_case(60, 36, max_iter=ITERS)
    batch = cases.product_batch(rq, case)
    good, bad = [0.31, 0.09], [0.95, 0.09]
    alone = batch.evaluate([good])
    for pattern in ("b", "bbb", "gb", "bg", "bbgbbbbg" * 30, "b" * 200, "g" + "b" * 150 + "g"):
        rows = batch.evaluate([good if ch == "g" else bad for ch in pattern]).rows
        for ch, row in zip(pattern, rows):
            if ch == "g":
                assert row.result.status == alone.rows[0].result.status
                np.testing.assert_array_equal(row.result.predictions, alone.predictions[0])
            else:
                assert row.result.status == rq.EvaluationStatus.InvalidParameters
                assert row.result.log_lik == -1e30


def test_eight_ctas(rq, checker):
    check_fields(rq, checker, cases.bump_case(260, 128, max_iter=3))


def test_more_cells_than_16_bit_columns(rq, checker):
    """From about 57 000 cells on, an inner tolerance of 1e-3 leaves so much of the pinned
    pressure mode open that two orders of the same sums differ by 1e-7 to 1e-4 after one outer
    iteration (one CTA of 512 against one of 768 threads, and either against the
    restatement). So the bound is ten times what the CTA sizes show on the same mesh."""
    case = cases.bump_case(330, 200, max_iter=2)
    want = checker.solve(case, "oracle")

    def distance(block):
        batch = cases.product_batch(rq, case, block_threads=block)
        res, fields, _ = batch.evaluate_fields([[case.coeffs[9], case.coeffs[8]]])
        assert res.rows[0].result.status.name == want.status
        return np.array([np.max(np.abs(fields[0, i] - want.fields[i])) /
                         max(np.max(np.abs(want.fields[i])), 1.0) for i in (0, 1, 3, 4, 5, 6, 7)])

    one = np.maximum(distance(512), distance(1024))
    assert np.all(one < 1e-3)
    assert np.all(distance(0) <= 10 * one + 1e-9)


@pytest.mark.parametrize("solver,precision", [("AMG", "fp64"), ("PCG", "fp64"),
                                              ("BiCGSTAB", "fp64"), ("AMG", "mixed"),
                                              ("BiCGSTAB", "mixed")])
@pytest.mark.parametrize("nx,ny", [(49, 32), (60, 36), (100, 50)])
def test_rows_do_not_depend_on_the_number_of_draws(rq, nx, ny, solver, precision):
    case = cases.bump_case(nx, ny, max_iter=8, turb_start=2)
    batch = cases.product_batch(rq, case, pressure_solver=solver, precision=precision)
    theta = np.array([[0.29, 0.085], [0.31, 0.09], [0.33, 0.095]])
    alone = [batch.evaluate_fields(theta[i:i + 1])[1][0] for i in range(3)]
    for n in (3, 40, 75, 160):  # 4, 2, 1 and 1 CTAs per solve on a B200
        _, fields, _ = batch.evaluate_fields(np.tile(theta, (n, 1))[:n])
        for i, f in enumerate(fields):
            np.testing.assert_array_equal(f, alone[i % 3])


@pytest.mark.parametrize("n", [20, 40, 70])  # 8, 4 and 2 CTAs
def test_rows_of_an_eight_cta_class(rq, n):
    case = cases.bump_case(260, 128, max_iter=3)
    batch = cases.product_batch(rq, case)
    want = batch.evaluate([[0.31, 0.09]]).predictions[0]
    for row in batch.evaluate(np.repeat([[0.31, 0.09]], n, axis=0)).predictions:
        np.testing.assert_array_equal(row, want)


def test_a_long_queue_fills_the_gpu(rq):
    """Enough draws for every SM run one per SM, not four or eight SMs each."""
    import torch
    from test_gpu_residency import most_at_once

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = cases.product_batch(rq, cases.bump_case(64, 40, max_iter=60))
    assert most_at_once(rq, batch, sms) >= 0.9 * sms


@pytest.mark.parametrize("nx,ny", [(60, 36), (100, 50)])
def test_results_do_not_depend_on_the_arena(rq, nx, ny):
    batch = cases.product_batch(rq, cases.bump_case(nx, ny, max_iter=8, turb_start=2))
    theta = np.array([[0.29, 0.085], [0.31, 0.09]])
    _, want, _ = batch.evaluate_fields(theta)
    for arena in (0, 40, 200):
        batch.set_launch(768, arena)
        _, got, _ = batch.evaluate_fields(theta)
        np.testing.assert_array_equal(got, want)
