"""k_bres (many steps per launch, the density on the chip) against the
per-step kernels on the same batches, every instance and its edges.

Tolerance: the two sides apply the same sums per cell and differ in the
order of the wake sums (N terms) and row sums only: below 4 eps = 2.4e-7 of
a value per step, 12 steps within 3e-6 relative L1; charges, averages over a
bunch, within 1e-6."""
import numpy as np
import pytest

from inovesa_gb300 import params as P
from inovesa_gb300 import vfps as V

pytestmark = pytest.mark.gpu


def rel_l1(a, b):
    b = np.asarray(b, np.float64)
    return float(np.abs(np.asarray(a, np.float64) - b).sum()
                 / np.abs(b).sum())


def batch(ctx, n, nb, it=4, renorm=0, wake=True, edit=None, spt=1000):
    p = P.derive(GridSize=n, StepsPerTs=spt, padding=2.0, S_csr=1.0,
                 RenormalizeCharge=renorm)
    z = V.makeImpedance(ctx, **P.wake_impedance_args(p))
    descs = []
    for s in np.linspace(0.1, 1.2, nb):
        d = P.fill_desc(V.BunchDesc(), p, 0,
                        Ib=p["I_norm"] * float(s) if wake else 0.0,
                        impedance=0, it=it)
        if edit:
            edit(d)
        descs.append(d)
    b = V.BunchBatch(ctx, descs, [z])
    rng = np.random.default_rng(n + nb)
    q = np.linspace(-6, 6, n)
    w = np.full(n, 2.0)
    w[1::2] = 4.0
    w[0] = w[-1] = 1.0
    w *= 12.0 / (n - 1) / 3.0
    out = []
    for i in range(nb):
        a = rng.uniform(-0.3, 0.3, size=3)
        d = np.exp(-0.5 * ((q[:, None] - a[0]) ** 2
                           + (q[None, :] - a[1]) ** 2))
        d *= 1 + 0.1 * np.sin(3 * q[:, None] + a[2])
        out.append(d / np.einsum("xy,x,y->", d, w, w))
    b.upload(np.concatenate([o.ravel() for o in out]).astype(np.float32))
    return b, p, z


def both(ctx, monkeypatch, steps, csr=False, **kw):
    res = []
    for env in (None, "steps"):
        if env:
            monkeypatch.setenv("VFPS_RING_KERNEL", env)
        b, p, z = batch(ctx, **kw)
        nb = len(b.descs)
        if csr:
            b.set_csr([z], [0] * nb, [p["fc"]] * nb, [P.C / p["bl"]] * nb,
                      every=2, capacity=4)
        for k in steps:
            b.step(k)
        out = [b.download(), b.profiles(), b.wake(), b.filling()]
        if csr:
            out += list(b.csr())
        res.append(out)
        monkeypatch.delenv("VFPS_RING_KERNEL", raising=False)
        assert ctx.device_status() == 0
    return res


def check(a, b):
    for x, y in zip(a[:2], b[:2]):
        assert rel_l1(x, y) <= 3e-6, rel_l1(x, y)
    if np.abs(b[2]).max() > 0:
        assert rel_l1(a[2], b[2]) <= 1e-5
    assert np.abs(a[3] - b[3]).max() <= 1e-6
    if len(a) > 4:
        assert np.array_equal(a[4], b[4])   # the recorded steps


# (mesh, bunches): every instance, and clusters with several bunches
@pytest.mark.parametrize("n,nb", [(64, 1), (64, 700), (128, 1), (128, 30),
                                  (128, 170), (256, 1), (256, 12), (256, 30),
                                  (256, 80)])
def test_instances(gpu_ctx, monkeypatch, n, nb):
    # single steps on either side of a long call (the step counters and
    # both buffers are shared with the per-step kernels)
    a, b = both(gpu_ctx, monkeypatch, (1, 10, 1), n=n, nb=nb)
    check(a, b)


@pytest.mark.parametrize("n,nb", [(64, 3), (128, 2), (128, 20), (256, 2)])
@pytest.mark.parametrize("it", [2, 3])
def test_orders(gpu_ctx, monkeypatch, n, nb, it):
    a, b = both(gpu_ctx, monkeypatch, (12,), n=n, nb=nb, it=it)
    check(a, b)


@pytest.mark.parametrize("n,nb", [(64, 2), (128, 2), (256, 2), (256, 30)])
def test_renormalisation_and_csr(gpu_ctx, monkeypatch, n, nb):
    a, b = both(gpu_ctx, monkeypatch, (5, 7), n=n, nb=nb, renorm=3, csr=True)
    check(a, b)


@pytest.mark.parametrize("n,nb", [(64, 2), (128, 2), (128, 20), (256, 2),
                                  (256, 12), (256, 30)])
def test_csr_power(gpu_ctx, n, nb):
    """The recorded power against 64 bits from the same profile.  The table
    K and the FP32 row sums (N / 32 products in sequence, 5 levels of a
    tree, the table's and the product's own roundings) are within
    (N / 32 + 7) eps / 2 of the sum of magnitudes |P| |K| |P|; the dot
    product over the rows is compensated."""
    b, p, z = batch(gpu_ctx, n, nb)
    b.set_csr([z], [0] * nb, [p["fc"]] * nb, [P.C / p["bl"]] * nb, every=15,
              capacity=1)
    b.step(15)
    prof = b.profiles().reshape(nb, n).astype(np.float64)
    # of the next 12 steps only the first (step 15) is recorded
    b.step(12)
    steps, power = b.csr()
    assert list(steps) == [15]
    zr = z.data().real.astype(np.float64)
    nmax = len(zr)
    dq = np.float64(np.float32((p["axes"][1] - p["axes"][0]) / (n - 1)))
    f = np.arange(nmax // 2 + 1)
    df = 1.0 / dq / (nmax - 1)
    c = dq * dq * zr[:nmax // 2 + 1] * (
        1 - np.exp(-(P.C / p["bl"] * df * f / p["fc"]) ** 2))
    d = np.arange(1 - n, n)
    K = df * (c[None, :] * np.cos(2 * np.pi * ((d[:, None] * f) % nmax)
                                  / nmax)).sum(1)
    T = K[np.arange(n)[:, None] - np.arange(n)[None, :] + n - 1]
    want = np.einsum("bx,xm,bm->b", prof, T, prof)
    mag = np.einsum("bx,xm,bm->b", abs(prof), abs(T), abs(prof))
    eps = 2.0 ** -23
    assert (np.abs(power[0] - want) <= (n / 32 + 7) * eps / 2 * mag).all()


@pytest.mark.parametrize("n,nb", [(64, 2), (256, 2)])
def test_without_wake(gpu_ctx, monkeypatch, n, nb):
    a, b = both(gpu_ctx, monkeypatch, (12,), n=n, nb=nb, wake=False)
    check(a, b)


@pytest.mark.parametrize("n,nb", [(64, 2), (128, 2), (256, 2), (256, 30)])
@pytest.mark.parametrize("angle", [0.05, 0.3, -0.3])
def test_far_kicks(gpu_ctx, monkeypatch, n, nb, angle):
    """RF kicks of up to 0.3 x n / 2 cells: windows at every alignment, past
    the zero words around a row and past the row's ends."""
    def edit(d):
        d.rf_angle = angle
    a, b = both(gpu_ctx, monkeypatch, (3,), n=n, nb=nb, edit=edit)
    check(a, b)


@pytest.mark.parametrize("n,nb", [(128, 2), (256, 2), (256, 30)])
def test_wide_drift(gpu_ctx, monkeypatch, n, nb):
    """A drift of several rows (edge rows of the neighbours on both sides)."""
    a, b = both(gpu_ctx, monkeypatch, (6,), n=n, nb=nb, spt=150)
    check(a, b)
