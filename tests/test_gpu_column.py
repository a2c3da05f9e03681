"""k_bcol (512-row meshes, many steps per launch) against the per-step kernels
on the same batches.

Tolerance: the two sides apply the same sums per cell and differ in the
order of the wake sums (512 terms) and row sums only: below 4 eps = 2.4e-7
of a value per step, 12 steps within 3e-6 relative L1; charges, averages
over a bunch, within 1e-6."""
import numpy as np
import pytest

from test_gpu_resident import both, check

pytestmark = pytest.mark.gpu


# one round of clusters and more than one; a call of many steps, of few
@pytest.mark.parametrize("nb", [1, 3, 9])
def test_bunches(gpu_ctx, monkeypatch, nb):
    check(*both(gpu_ctx, monkeypatch, (11, 1), n=512, nb=nb))


@pytest.mark.parametrize("it", [2, 3])
def test_orders(gpu_ctx, monkeypatch, it):
    check(*both(gpu_ctx, monkeypatch, (12,), n=512, nb=2, it=it))


def test_renormalisation_and_csr(gpu_ctx, monkeypatch):
    check(*both(gpu_ctx, monkeypatch, (12,), csr=True, n=512, nb=2,
                renorm=3))


def test_without_wake(gpu_ctx, monkeypatch):
    check(*both(gpu_ctx, monkeypatch, (12,), n=512, nb=2, wake=False))


# kicks past the zero lines around the density (rows of any shift), rows
# kicked off the mesh
@pytest.mark.parametrize("angle", [0.05, 0.4, 2.0])
def test_far_kicks(gpu_ctx, monkeypatch, angle):
    def edit(d):
        d.rf_angle = angle
    check(*both(gpu_ctx, monkeypatch, (12,), n=512, nb=2, spt=4000,
                edit=edit))


# a drift of more than two rows stays on the per-step kernels
def test_wide_drift(gpu_ctx, monkeypatch):
    check(*both(gpu_ctx, monkeypatch, (12,), n=512, nb=2, spt=400))
