"""One batched step of the rotation chain against the 64-bit maps, for every
mesh size, interpolation order and clamping, with small and large angles and
kicks (tiles whose source rows jump, rows kicked past the mesh).

Tolerance: a source coordinate (a sum of products, about 4 roundings of a
value up to n) is off by at most 4 * 6e-8 * n cells, which moves a density of
gradient 12 / n per cell by 3e-6 of itself at most; the weights, taps and
the two maps after it add about 20 roundings of 6e-8 each.  Relative L1
within 5e-6; each bunch's profile sums the same cells, within 5e-6 too."""
import numpy as np
import pytest

import oracle
from inovesa_gb300 import params as P
from inovesa_gb300 import vfps as V
from inovesa_gb300._lib import InvalidArgument

pytestmark = pytest.mark.gpu

NB = 3


def simpson(n, width):
    w = np.full(n, 2.0)
    w[1::2] = 4.0
    w[0] = w[-1] = 1.0
    return w * width / (n - 1) / 3.0


def rel_l1(a, b):
    return float(np.abs(np.asarray(a, np.float64) - b).sum()
                 / np.abs(b).sum())


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024])
@pytest.mark.parametrize("it,clamp", [(2, False), (3, False), (4, False),
                                      (4, True)])
@pytest.mark.parametrize("angle,current", [(0.006, 1.0), (0.05, 1.0),
                                           (0.006, 4000.0)])
def test_step(gpu_ctx, n, it, clamp, angle, current):
    p = P.derive(GridSize=n, StepsPerTs=1000, padding=2.0, S_csr=1.0,
                 RenormalizeCharge=0)
    axes = tuple(p["axes"])
    z = V.makeImpedance(gpu_ctx, **P.wake_impedance_args(p))
    descs = []
    for s in np.linspace(0.3, 1.2, NB):
        d = P.fill_desc(V.BunchDesc(), p, 1, Ib=p["I_norm"] * s * current,
                        impedance=0, it=it, clamp=clamp)
        d.angle = angle
        descs.append(d)
    q = np.linspace(axes[0], axes[1], n)
    rho = np.exp(-0.5 * ((q[None, :, None] - 0.3) ** 2
                         + (q[None, None, :] + 0.2) ** 2))
    rho = rho * (1 + 0.2 * np.sin(q[None, :, None] * (1 + np.arange(NB))[
        :, None, None] + 0.7 * q[None, None, :]))
    ws = simpson(n, axes[1] - axes[0])
    rho /= np.einsum("bxy,x,y->b", rho, ws, ws)[:, None, None]
    rho = rho.astype(np.float32)
    if n == 1024 and angle == 0.05:
        # 26 source rows on either side of a tile: more than fits on the chip
        with pytest.raises(InvalidArgument):
            V.BunchBatch(gpu_ctx, descs, [z])
        return
    b = V.BunchBatch(gpu_ctx, descs, [z])
    b.upload(rho.ravel())
    b.step(1)
    got = np.asarray(b.download()).reshape(NB, n, n)
    wake = np.asarray(b.wake()).reshape(NB, n)
    prof = np.asarray(b.profiles()).reshape(NB, n)
    assert gpu_ctx.device_status() == 0
    idx, w = oracle.fp_stencils(n, axes, descs[0].e1, descs[0].fptype,
                                descs[0].derivation, dtype=np.float64)
    for i in range(NB):
        ref = oracle.rotation(rho[i:i + 1], axes, angle, it, clamp)
        ref = oracle.kick(1, ref, it, wake[i].astype(np.float64))
        ref = oracle.fp_apply(ref, descs[0].derivation, idx, w)[0]
        assert rel_l1(got[i], ref) <= 5e-6
        assert rel_l1(prof[i], ref @ ws) <= 5e-6
