"""A bunch's state is the same to the bit however a run is cut into calls,
whichever kernels its calls take (k_bres, k_bcol or a launch per step,
k_bmaps0f or k_bstrip) and whatever other bunches the batch holds."""
import numpy as np
import pytest

from inovesa_gb300 import params as P
from inovesa_gb300 import vfps as V
from test_gpu_routes import two_rounds_512

pytestmark = pytest.mark.gpu


class Bunch:
    """(mesh, order, steps per period, seed) of a bunch."""

    def __init__(self, n, it=4, spt=4000, seed=0, renorm=3):
        self.n, self.it, self.seed = n, it, seed
        self.p = P.derive(GridSize=n, StepsPerTs=spt, padding=2.0, S_csr=1.0,
                          RenormalizeCharge=renorm)
        self.key = (n, spt, renorm)

    def density(self):
        r = np.random.default_rng([self.n, self.seed])
        a = r.uniform(-0.3, 0.3, size=3)
        q = np.linspace(-6, 6, self.n)
        d = np.exp(-0.5 * ((q[:, None] - a[0]) ** 2
                           + (q[None, :] - a[1]) ** 2))
        d *= 1 + 0.1 * np.sin(3 * q[:, None] + a[2])
        return (d / (d.sum() * (q[1] - q[0]) ** 2)).astype(np.float32)


def run(ctx, bunches, calls, csr=True, wake=True):
    """State of every bunch after the calls ("t": through kernel_times)."""
    zs = {}
    for b in bunches:
        if b.key not in zs:
            zs[b.key] = (len(zs), V.makeImpedance(
                ctx, **P.wake_impedance_args(b.p)))
    descs = [P.fill_desc(V.BunchDesc(), b.p, 0,
                         Ib=b.p["I_norm"] * (0.2 + 0.07 * b.seed)
                         if wake else 0.0,
                         impedance=zs[b.key][0], it=b.it) for b in bunches]
    zl = [z for _, z in zs.values()]
    m = V.BunchBatch(ctx, descs, zl)
    m.upload(np.concatenate([b.density().ravel() for b in bunches]))
    if csr:
        m.set_csr(zl, [zs[b.key][0] for b in bunches],
                  [b.p["fc"] for b in bunches],
                  [P.C / b.p["bl"] for b in bunches], every=2, capacity=16)
    for c in calls:
        if isinstance(c, str):
            m.kernel_times(int(c))
        else:
            m.step(c)
    assert ctx.device_status() == 0
    dens, prof, wk, fill = m.download(), m.profiles(), m.wake(), m.filling()
    power = m.csr()[1] if csr else np.zeros((1, len(bunches)))
    out = []
    for i, b in enumerate(bunches):
        d, r = m.layout(i)
        n = b.n
        out.append((dens[d:d + n * n], prof[r:r + n], wk[r:r + n],
                    fill[i], power[:, i]))
    return m, out


def same(a, b):
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            assert np.array_equal(u, v), np.abs(u - v).max()


# (mesh, steps a period, bunches): every instance and several rounds
# (the last: as many bunches as two rounds of k_bcol's clusters take)
KINDS = [(64, 4000, 1), (64, 1000, 700), (128, 1000, 1), (128, 1000, 30),
         (128, 201, 170), (256, 1000, 1), (256, 4000, 12), (256, 201, 30),
         (256, 1000, 80), (512, 4000, 1), (512, 4000, 0)]


@pytest.mark.parametrize("n,spt,nb", KINDS)
@pytest.mark.parametrize("it", [2, 4])
def test_calls(gpu_ctx, monkeypatch, n, spt, nb, it):
    bunches = [Bunch(n, it, spt, s % 16)
               for s in range(nb or two_rounds_512(gpu_ctx))]
    monkeypatch.setenv("VFPS_RING_KERNEL", "steps")
    m, want = run(gpu_ctx, bunches, [1] * 23)
    assert not m.route(23)["resident"]
    monkeypatch.delenv("VFPS_RING_KERNEL")
    for calls in ((23,), (12, 1, 10), ("11", 12)):
        m, got = run(gpu_ctx, bunches, calls)
        assert m.route(12)["resident"]
        same(got, want)


@pytest.mark.parametrize("n,nb", [(128, 2), (256, 2), (512, 2)])
def test_calls_without_wake(gpu_ctx, monkeypatch, n, nb):
    bunches = [Bunch(n, 3, 4000, s, renorm=0) for s in range(nb)]
    monkeypatch.setenv("VFPS_RING_KERNEL", "steps")
    _, want = run(gpu_ctx, bunches, [1] * 9, csr=False, wake=False)
    monkeypatch.delenv("VFPS_RING_KERNEL")
    m, got = run(gpu_ctx, bunches, (9,), csr=False, wake=False)
    assert m.route(9)["resident"]
    same(got, want)


# the same bunches alone, among many of their mesh, beside a mesh that keeps
# the whole batch on the per-step kernels, beside a lattice that is not regular
@pytest.mark.parametrize("n,spt", [(64, 1000), (128, 1000), (256, 1000),
                                   (512, 4000)])
def test_company(gpu_ctx, n, spt):
    mine = [Bunch(n, 4, spt, s) for s in range(2)]
    m, want = run(gpu_ctx, mine, (13,))
    assert m.route(13)["resident"]
    others = [
        [Bunch(n, 4, spt, s % 16) for s in range(2, 90 if n < 512 else 13)],
        [Bunch(1024, 4, 4000, 3)],
        [Bunch(64, 3, 90, 1), Bunch(512, 2, 700, 4)],
    ]
    for o in others:
        _, got = run(gpu_ctx, mine + o, (13,))
        same(got[:2], want)


# a launch per step: the kernels of wide meshes that the autotuner picks from
@pytest.mark.parametrize("n,spt", [(512, 4000), (512, 2000), (1024, 4000),
                                   (1024, 2000)])
@pytest.mark.parametrize("it", [2, 3, 4])
def test_wide_kernels(gpu_ctx, monkeypatch, n, spt, it):
    bunches = [Bunch(n, it, spt, s) for s in range(3)]
    out = []
    for tile, kernel in (("2000", "steps"), ("8000", "steps"),
                         ("900", "strips"), ("8000", "strips"),
                         ("13200", "strips")):
        monkeypatch.setenv("VFPS_RING_KERNEL", kernel)
        monkeypatch.setenv("VFPS_TILE_CELLS", tile)
        m, got = run(gpu_ctx, bunches, (7,))
        assert not m.route(7)["resident"]
        out.append(got)
    for got in out[1:]:
        same(got, out[0])
