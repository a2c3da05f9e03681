"""The potential-well start with one to eight CTAs per bunch (chosen by the
number of bunches): the same operations in the same order, so the same bits
for the same bunch in batches of any size."""
import numpy as np
import pytest

from test_gpu_potential_well import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,counts", [(64, (1, 90, 160)),
                                      (256, (1, 17, 64, 160)),
                                      (512, (1, 30, 100))])
def test_same_state(gpu_ctx, n, counts):
    want = None
    for nb in counts:
        b, _ = batch(gpu_ctx, [(n, 0.30, 0.006, 0, True)] * nb, spt=4000)
        b.potential_well(iterations=7, mix=0.5)
        for i in (0, nb - 1):
            got = b.density(i)
            want = got if want is None else want
            assert np.array_equal(got, want)
        assert gpu_ctx.device_status() == 0
