"""Densities that are not finite spread through the Fokker-Planck map's row
sweeps exactly as through its thread-per-cell kernel: one NaN or infinity per
row, in the columns at the edges, next to them and inside.  (The columns at
the edges have no stencil: they are column 0 times 0, as in the reference.)"""
import numpy as np
import pytest

from inovesa_gb300 import vfps as V
from test_gpu_plain_rows import density, pair, use_cells

pytestmark = pytest.mark.gpu


def spoiled(n):
    d = density(n, 2, seed=n)
    at = [0, 1, 2, 3, n // 2, n - 4, n - 3, n - 2, n - 1]
    for k, p in enumerate(at):
        v = (np.nan, np.inf, -np.inf)[k % 3]
        d[k % 2, 2 * k + 5, p] = v
    return d


@pytest.mark.parametrize("n", [64, 256])
@pytest.mark.parametrize("derivation", [3, 4])
@pytest.mark.parametrize("fptype", [0, 3])
def test_fokker_planck(gpu_ctx, monkeypatch, n, derivation, fptype):
    d, out = spoiled(n), []
    for cells in (False, True):
        use_cells(monkeypatch, cells)
        a, b = pair(gpu_ctx, n, d)
        a.setData(d)
        V.FokkerPlanckMap(a, b, n, n, fptype, 0, 2e-3, derivation).apply()
        out.append(b.getData())
    np.testing.assert_array_equal(out[0], out[1])
    assert np.isnan(out[0]).any()
    gpu_ctx.device_status()
