"""Batches that live at the same time do not disturb one another: a batch
made later, with smaller tiles and other kernels, leaves the calls of an
earlier one as they were (vfps_batch_run in parts and vfps_batch_kernel_times
launch the per-step kernels directly, not through the captured graphs)."""
import numpy as np
import pytest
import torch

from inovesa_gb300 import params as P
from inovesa_gb300 import vfps as V

pytestmark = pytest.mark.gpu


def batch(ctx, kinds):
    """kinds: (mesh, chain, order) of each bunch."""
    ps = {n: P.derive(GridSize=n, StepsPerTs=2000, padding=2.0, S_csr=1.0)
          for n, _, _ in kinds}
    zs = {n: (i, V.makeImpedance(ctx, **P.wake_impedance_args(p)))
          for i, (n, p) in enumerate(ps.items())}
    descs = [P.fill_desc(V.BunchDesc(), ps[n], chain,
                         Ib=ps[n]["I_norm"] * 0.5, impedance=zs[n][0], it=it)
             for n, chain, it in kinds]
    return V.BunchBatch(ctx, descs, [z for _, z in zs.values()])


@pytest.mark.parametrize("kinds", [
    [(256, 1, 4)] * 161,
    [(1024, 0, 4)] * 12,
    [(1024, 0, 3), (512, 0, 2), (256, 0, 4), (128, 1, 3), (64, 0, 4)] * 14,
])
def test_a_smaller_batch_beside(gpu_ctx, monkeypatch, kinds):
    monkeypatch.setenv("VFPS_TILE_CELLS", "8192")
    a = batch(gpu_ctx, kinds)
    start = a.download()
    out = torch.zeros(a.cells, dtype=torch.float32, pin_memory=True).numpy()
    a.run(start, 12, out)
    want = out.copy()
    monkeypatch.setenv("VFPS_TILE_CELLS", "1024")
    b = batch(gpu_ctx, [(64, 0, 4), (64, 1, 4)])
    b.step(2)
    a.run(start, 12, out)
    assert np.array_equal(out, want)
    a.kernel_times(2)
    assert gpu_ctx.device_status() == 0
