"""vfps_batch_run into page-locked memory copies parts of the batch while
others are computed: the same bytes as the steps and the copy one after the
other, for bunches that fill one round of clusters, several, and leave some
over; and for the calls that keep the single copy (small batches, ordinary
memory, several mesh sizes)."""
import numpy as np
import pytest
import torch

from test_gpu_resident import batch

pytestmark = pytest.mark.gpu


def run(ctx, n, nb, steps, pinned):
    b, p, z = batch(ctx, n=n, nb=nb)
    t = torch.zeros(b.cells, dtype=torch.float32, pin_memory=pinned)
    prof = np.zeros(b.rows, np.float32)
    fill = np.zeros(nb, np.float32)
    for k in steps:
        b.run(None, k, t.numpy(), prof, fill)
    assert ctx.device_status() == 0
    assert np.array_equal(t.numpy(), b.download())
    return t.numpy().copy(), prof, fill, b.wake()


@pytest.mark.parametrize("n,nb", [(64, 700), (128, 30), (128, 170),
                                  (256, 40), (256, 80), (512, 9)])
def test_same_bytes(gpu_ctx, n, nb):
    a = run(gpu_ctx, n, nb, (30, 31), True)
    b = run(gpu_ctx, n, nb, (30, 31), False)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
