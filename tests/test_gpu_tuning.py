"""The tile size that one batch found best is for batches like it: the same
meshes with the same kernels to choose from."""
import pytest

from inovesa_gb300 import vfps as V
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


@pytest.mark.parametrize("cells", [1 << 24, (1 << 24) + 8192])
def test_forced_size_is_a_size(gpu_ctx, monkeypatch, cells):
    """A forced tile of whole 1024-row meshes does not fit on the chip,
    whatever bits its size has."""
    monkeypatch.setenv("VFPS_TILE_CELLS", str(cells))
    with pytest.raises(V.VfpsError):
        batch(gpu_ctx, n=1024, nb=1, spt=4000)
