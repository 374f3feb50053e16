"""How many draws run at once, from the solves' own start and end stamps: CTAs of fewer than
512 threads leave registers for a second one, and where draws wait their default arena leaves
it shared memory. Results do not depend on the arena."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def most_at_once(rq, batch, n):
    import torch

    dev = torch.device("cuda", 0)
    th = torch.tensor(np.repeat([[0.31, 0.09]], n, axis=0), dtype=torch.float64, device=dev)
    rows = torch.zeros(n * 40, dtype=torch.uint8, device=dev)
    pred = torch.zeros((n, 8), dtype=torch.float64, device=dev)
    clock = torch.zeros((n, 12), dtype=torch.int64, device=dev)
    for _ in range(2):  # the first launch also loads the kernel
        rq.evaluate_multi_device([batch], np.zeros(n, dtype=np.int32), th.data_ptr(),
                                 rows.data_ptr(), pred.data_ptr(),
                                 torch.cuda.current_stream(dev).cuda_stream, clock.data_ptr())
        torch.cuda.synchronize()
    ck = clock.cpu().numpy()
    return max(int(np.sum((ck[:, 0] <= t) & (ck[:, 1] > t))) for t in ck[:, 0])


@pytest.mark.parametrize("ny", [24, 128])
@pytest.mark.parametrize("block,per_sm", [(64, 2), (128, 2), (256, 2), (512, 1)])
def test_draws_per_sm(rq, ny, block, per_sm):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = cases.product_batch(rq, cases.small_channel(ny=ny, max_iter=200), block_threads=block)
    at_once = most_at_once(rq, batch, 2 * sms)
    assert at_once >= 0.9 * per_sm * sms


@pytest.mark.parametrize("ny,block", [(24, 64), (24, 512), (128, 128), (128, 256), (128, 512),
                                      (300, 512), (512, 512), (513, 512)])
def test_results_do_not_depend_on_the_arena(rq, ny, block):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = cases.product_batch(rq, cases.small_channel(ny=ny, max_iter=12, turb_start=2))
    theta = np.array([[0.29, 0.085], [0.31, 0.09], [0.33, 0.095]])
    batch.set_launch(block, -1)
    want, fields, _ = batch.evaluate_fields(theta)
    many = batch.evaluate(np.concatenate([theta] * (sms // 3 + 1))).predictions
    for i, row in enumerate(many):
        np.testing.assert_array_equal(row, want.predictions[i % 3])
    for arena in (0, 20, 100, 200):
        batch.set_launch(block, arena)
        _, got, _ = batch.evaluate_fields(theta)
        np.testing.assert_array_equal(got, fields)
