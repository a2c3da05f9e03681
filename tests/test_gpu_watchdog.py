"""The charge watchdog (VFPS_ERR_NUMERIC) in the middle of a call that stays
on the chip: it goes by the compensated Simpson integral of every step, as the
per-step kernels do, whatever the profile looks like."""
import numpy as np
import pytest

from inovesa_gb300 import _lib
from test_gpu_resident import batch

pytestmark = pytest.mark.gpu

STEPS = 9


def rows_of(n, values):
    """Densities whose rows x hold values[x], spread over the energy axis."""
    q = np.linspace(-6, 6, n)
    d = np.zeros((n, n), np.float32)
    for x, v in values.items():
        d[x] = v * np.exp(-0.5 * q * q)
    return d


def status(ctx, monkeypatch, n, nb, density, kernel=None):
    if kernel:
        monkeypatch.setenv("VFPS_RING_KERNEL", kernel)
    b, _, _ = batch(ctx, n=n, nb=nb, wake=False, spt=4000)
    monkeypatch.delenv("VFPS_RING_KERNEL", raising=False)
    assert b.route(STEPS)["resident"] == (kernel is None)
    good = b.download()
    b.upload(np.tile(density.ravel(), nb))
    ctx.device_status()      # (the upload integrates too)
    b.step(STEPS)
    got = ctx.device_status()
    b.upload(good)
    b.step(STEPS)
    assert ctx.device_status() == 0
    return got


MESHES = [(64, 2), (128, 2), (128, 30), (256, 2), (256, 30), (512, 2)]


# The charge in units of two thirds of a cell: sums without the edge rows'
# half weights would call these the other way round.
@pytest.mark.parametrize("n,nb", MESHES)
def test_edge_rows(gpu_ctx, monkeypatch, n, nb):
    for values, want in (
            ({0: -1.0, 4: 0.75}, 0),                    # -0.5 + 0.75
            ({0: 1.0, 4: -0.75}, _lib.VFPS_ERR_NUMERIC),
            ({n - 1: -1.0, n - 6: 1.2}, 0),             # -0.5 + 1.2
            ({n - 1: 1.0, n - 6: -0.6}, _lib.VFPS_ERR_NUMERIC)):
        d = rows_of(n, values)
        assert status(gpu_ctx, monkeypatch, n, nb, d) == want, values
        assert status(gpu_ctx, monkeypatch, n, nb, d, "steps") == want


@pytest.mark.parametrize("n,nb", MESHES)
@pytest.mark.parametrize("value", [0.0, np.nan, np.inf, -np.inf])
def test_no_charge(gpu_ctx, monkeypatch, n, nb, value):
    d = rows_of(n, {n // 2: value, n // 2 + 1: value})
    for kernel in (None, "steps"):
        assert status(gpu_ctx, monkeypatch, n, nb, d, kernel) \
            == _lib.VFPS_ERR_NUMERIC


# a charge of 4e-6 of the profile's magnitude: two even rows that nearly cancel
# (an FP32 sum alone would not be trusted with its sign)
@pytest.mark.parametrize("n,nb", MESHES)
@pytest.mark.parametrize("sign", [1, -1])
def test_small_charge(gpu_ctx, monkeypatch, n, nb, sign):
    d = rows_of(n, {n // 2: 1.0, n // 2 + 2: -1.0 + sign * 8e-6})
    want = 0 if sign > 0 else _lib.VFPS_ERR_NUMERIC
    for kernel in (None, "steps"):
        assert status(gpu_ctx, monkeypatch, n, nb, d, kernel) == want
