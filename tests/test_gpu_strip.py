"""k_bstrip (512- and 1024-row meshes, one step per launch) against the
general per-step kernels on the same batches: every order, tiles of few and
many rows, narrow and wide drifts, kicks of any size.

Tolerance: the general kernels apply the two y-kicks as one or two stencils
with the same weights and add the row sums in another order: below 8 eps =
5e-7 of a value per step, 6 steps within 3e-6 relative L1; charges, averages
over a bunch, within 1e-6."""
import numpy as np
import pytest

from test_gpu_resident import batch, rel_l1

pytestmark = pytest.mark.gpu


def sides(ctx, monkeypatch, tile=None, **kw):
    out = []
    for kernel in ("strips", "classic"):
        monkeypatch.setenv("VFPS_RING_KERNEL", kernel)
        if tile and kernel == "strips":
            monkeypatch.setenv("VFPS_TILE_CELLS", str(tile))
        b, p, z = batch(ctx, **kw)
        b.step(6)
        out.append([b.download(), b.profiles(), b.filling()])
        monkeypatch.delenv("VFPS_TILE_CELLS", raising=False)
        assert ctx.device_status() == 0
    (d, p, f), (dr, pr, fr) = out
    assert rel_l1(d, dr) <= 3e-6, rel_l1(d, dr)
    assert rel_l1(p, pr) <= 3e-6, rel_l1(p, pr)
    assert np.abs(f - fr).max() <= 1e-6


@pytest.mark.parametrize("n", [512, 1024])
@pytest.mark.parametrize("it", [2, 3, 4])
def test_orders(gpu_ctx, monkeypatch, n, it):
    sides(gpu_ctx, monkeypatch, n=n, nb=2, it=it, spt=4000)


# a tile of 4 rows, of a number that leaves a remainder, of the most rows
@pytest.mark.parametrize("n", [512, 1024])
@pytest.mark.parametrize("tile", [500, 8000, 13200])
def test_tiles(gpu_ctx, monkeypatch, n, tile):
    sides(gpu_ctx, monkeypatch, tile=tile, n=n, nb=3, spt=4000, renorm=2)


# drifts of up to 2, 4 and 8 rows at the ends of the energy axis
# (past 800 steps a period the general kernel's tile of 1024 rows does not
# fit on the chip)
@pytest.mark.parametrize("n,spt", [(512, 2000), (512, 800), (512, 500),
                                   (1024, 2000), (1024, 800)])
def test_drifts(gpu_ctx, monkeypatch, n, spt):
    sides(gpu_ctx, monkeypatch, n=n, nb=2, spt=spt)


@pytest.mark.parametrize("n", [512, 1024])
@pytest.mark.parametrize("angle", [0.05, 0.4, 2.0])
def test_far_kicks(gpu_ctx, monkeypatch, n, angle):
    def edit(d):
        d.rf_angle = angle
    sides(gpu_ctx, monkeypatch, n=n, nb=2, spt=4000, edit=edit)


# Lattices that are not regular: a strong wake and an opposite RF kick, with
# density up to the ends of the energy axis.  What the first kick moves off
# the axis does not come back with the second, on k_bstrip as on the general
# kernel: after one step from the same profile (the same wake to the bit)
# cells are within 64 eps of the largest (some ten roundings per cell, kicks
# with weights of up to 1.3 in sum).
@pytest.mark.parametrize("it", [2, 3, 4])
@pytest.mark.parametrize("spt,angle", [(700, 0.045), (700, -0.045),
                                       (500, 0.02), (600, 0.06)])
def test_kicks_in_turn(gpu_ctx, monkeypatch, it, spt, angle):
    n, out = 512, []

    def edit(d):
        d.rf_angle = angle
        d.wakescaling *= 200.0
    q = np.linspace(-1, 1, n)
    dens = np.outer(np.exp(-8 * q * q), 1 + 0.5 * np.cos(9 * q))
    w = np.full(n, 2.0)
    w[1::2] = 4.0
    w[0] = w[-1] = 1.0
    w *= 12.0 / (n - 1) / 3.0
    dens = np.tile((dens / (w @ dens @ w)).astype(np.float32).ravel(), 2)
    for kernel in ("strips", "classic"):
        monkeypatch.setenv("VFPS_RING_KERNEL", kernel)
        b, _, _ = batch(gpu_ctx, n=n, nb=2, it=it, spt=spt, edit=edit)
        tiles = b.kernel_tiles()
        # (a shift of more than 13 columns stays on the general kernel)
        on_strips = kernel == "strips" and abs(angle) < 0.05
        assert (tiles["k_bmaps0f"] > 0) == on_strips, tiles
        b.upload(dens)
        b.step(1)
        out.append((b.download(), b.wake()))
    (x, wx), (y, wy) = out
    assert np.array_equal(wx, wy) and 1.0 < np.abs(wx).max() < 60.0
    assert np.abs(x - y).max() <= 64 * 2.0 ** -23 * np.abs(y).max()
