"""vfps_batch_run into page-locked memory copies parts of the batch while
others are computed: the same bytes as the steps and the copy one after the
other, for bunches that fill one round of clusters, several, and leave some
over; and for the calls that keep the single copy (small batches, ordinary
memory, several mesh sizes)."""
import numpy as np
import pytest
import torch

from inovesa_gb300 import params as P
from inovesa_gb300 import vfps as V
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


def mixed(ctx, kinds, steps, pinned):
    """kinds: (mesh, chain, order) of each bunch."""
    ps = {n: P.derive(GridSize=n, StepsPerTs=2000, padding=2.0, S_csr=1.0,
                      RenormalizeCharge=0) for n, _, _ in kinds}
    index, zs = {}, []
    for n, p in ps.items():
        index[n] = len(zs)
        zs.append(V.makeImpedance(ctx, **P.wake_impedance_args(p)))
    descs = [P.fill_desc(V.BunchDesc(), ps[n], chain,
                         Ib=ps[n]["I_norm"] * (0.2 + 0.01 * i),
                         impedance=index[n], it=it)
             for i, (n, chain, it) in enumerate(kinds)]
    b = V.BunchBatch(ctx, descs, zs)
    t = torch.zeros(b.cells, dtype=torch.float32, pin_memory=pinned)
    prof = np.zeros(b.rows, np.float32)
    fill = np.zeros(len(kinds), np.float32)
    for k in steps:
        b.run(None, k, t.numpy(), prof, fill)
    assert ctx.device_status() == 0
    assert np.array_equal(t.numpy(), b.download())
    return t.numpy().copy(), prof, fill, b.wake()


# one kind (halves), several in turn, a batch whose parts would cost more than
# they save, calls shorter and longer than the part that runs apart
@pytest.mark.parametrize("kinds", [
    [(256, 1, 4)] * 161,
    [(1024, 0, 4)] * 12,
    [(512, 0, 3)] * 16,
    [(1024, 0, 3), (512, 0, 2), (256, 0, 4), (128, 1, 3), (64, 0, 4)] * 14,
    [(512, 0, 4), (256, 1, 2)] * 60,
])
@pytest.mark.parametrize("steps", [(1, 2), (3, 40)])
def test_same_bytes_per_step(gpu_ctx, kinds, steps):
    a = mixed(gpu_ctx, kinds, steps, True)
    b = mixed(gpu_ctx, kinds, steps, False)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
