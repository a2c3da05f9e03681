"""The tile size that one batch found best is for batches like it: the same
meshes with the same kernels to choose from."""
import pytest

from test_gpu_resident import batch

pytestmark = pytest.mark.gpu


def test_kernel_choice_is_part_of_the_key(gpu_ctx, monkeypatch):
    """24 bunches of 1024 rows take k_bstrip (55 us a step, 71 on k_bmaps0f),
    whose tiles have 14 rows or more, also after a batch of the same meshes
    was tuned with no choice of kernel (a size of k_bmaps0f's, whose tiles
    have 12 rows at most)."""
    kw = dict(n=1024, nb=24, spt=3917)
    monkeypatch.setenv("VFPS_RING_KERNEL", "strips")
    a, _, _ = batch(gpu_ctx, **kw)
    a.step(1)
    monkeypatch.delenv("VFPS_RING_KERNEL")
    b, _, _ = batch(gpu_ctx, **kw)
    assert b.info()[1] >= 14, b.info()
    b.step(3)
    assert gpu_ctx.device_status() == 0
