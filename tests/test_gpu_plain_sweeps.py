"""The plain path's kernels at the sizes where their splits can go wrong:
rows per thread of the rotation, column blocks and row blocks of the x-kick
and Fokker-Planck sweeps, the energy projection's 32 x 32 cut, warps per
bunch of the charge integral, runs of 16 cells of the CSR sum, the wake
table in and out of shared memory.

Tolerances: maps within 2e-6 of the largest value of the float restatement
(the order of operations is the same); projections, integrals and the CSR
power add FP32 products in FP64 after at most 32 of them: 32 eps / 2 =
2e-6 of the sum of magnitudes, positive terms for the first two; wake and
spectrum relative to their largest value, with the FP32 impedance sums'
cancellation of up to 10 allowed for (2e-5)."""
import math

import numpy as np
import pytest

import oracle
from inovesa_gb300 import vfps as V

pytestmark = pytest.mark.gpu

AXES = (-6.0, 6.0, 2e-3, -6.0, 6.0, 6.11e5)


def density(n, nb=1, seed=0):
    rng = np.random.default_rng(seed)
    q = np.linspace(-6, 6, n)
    out = []
    for b in range(nb):
        g = np.exp(-0.5 * (q[:, None] ** 2 + (q[None, :] - 0.3 + 0.1 * b)
                           ** 2))
        g *= 1 + 0.2 * np.sin(q[:, None] + 0.7 * q[None, :])
        g += 1e-3 * rng.random((n, n))
        out.append(g / g.sum() / nb)
    return np.stack(out).astype(np.float32)


def space(ctx, n, data):
    nb = len(data)
    return V.PhaseSpace(*AXES, ctx, 1, 1, [1.0 / nb] * nb, 1.0, data, n=n)


def simpson(n):
    w = np.full(n, 2.0)
    w[1::2] = 4.0
    w[0] = w[-1] = 1.0
    return w * 12.0 / (n - 1) / 3.0


@pytest.mark.parametrize("n,it,clamp", [(129, 4, True), (129, 1, False),
                                        (1030, 4, True), (1030, 4, False),
                                        (1030, 3, False), (1030, 2, False)])
def test_rotation(gpu_ctx, n, it, clamp):
    d = density(n, seed=n)
    a, b = space(gpu_ctx, n, d), space(gpu_ctx, n, d)
    for angle in (2 * math.pi / 700, 0.4):   # bases in order, and not
        V.RotationMap(a, b, n, n, angle, it, clamp,
                      n * n if clamp else 0).apply()
        ref = oracle.rotation(d, AXES, angle, it, clamp, dtype=np.float32)
        assert np.abs(b.getData() - ref).max() <= 2e-6 * np.abs(ref).max()


@pytest.mark.parametrize("n,nb", [(100, 3), (516, 3), (2052, 1)])
@pytest.mark.parametrize("it", [1, 2, 3, 4])
def test_x_kick(gpu_ctx, n, nb, it):
    d = density(n, nb, seed=it)
    a, b = space(gpu_ctx, n, d), space(gpu_ctx, n, d)
    k = V.KickMap(a, b, it, False, V.Axis.x)
    # shifts alike in groups of 4 columns, and not; some off the mesh
    for off in (np.repeat(np.linspace(-0.6 * n, 0.6 * n, n // 4), 4),
                np.linspace(-20, 20, n)):
        off = off.astype(np.float32)
        k.swapOffset(off)
        k.apply()
        ref = oracle.kick(0, d, it, off, dtype=np.float32)
        assert np.abs(b.getData() - ref).max() <= 2e-6 * np.abs(ref).max()


@pytest.mark.parametrize("n,nb", [(100, 3), (516, 3), (2052, 1)])
@pytest.mark.parametrize("dt", [3, 4])
def test_fokker_planck(gpu_ctx, n, nb, dt):
    d = density(n, nb, seed=dt)
    a, b = space(gpu_ctx, n, d), space(gpu_ctx, n, d)
    V.FokkerPlanckMap(a, b, n, n, 3, 0, 1e-6, dt).apply()
    idx, w = oracle.fp_stencils(n, AXES, 1e-6, 3, dt, dtype=np.float32)
    ref = oracle.fp_apply(d, dt, idx, w, dtype=np.float32)
    assert np.abs(b.getData() - ref).max() <= 2e-6 * np.abs(ref).max()


@pytest.mark.parametrize("n,nb", [(31, 1), (33, 2), (256, 3), (257, 5),
                                  (1000, 9)])
def test_projections_and_integral(gpu_ctx, n, nb):
    d = density(n, nb, seed=nb)
    a = space(gpu_ctx, n, d)
    a.updateXProjection()
    a.updateYProjection()
    a.integrate()
    w = simpson(n)
    x = d.astype(np.float64)
    px, py = x @ w, np.einsum("bxy,x->by", x, w)
    for got, want in ((a.getProjection(0), px), (a.getProjection(1), py)):
        assert (np.abs(got - want) <= 2e-6 * want).all()
    f = px @ w
    assert (np.abs(a.getBunchPopulation() - f) <= 2e-6 * f).all()
    assert abs(a.getIntegral() - f.sum()) <= 2e-6 * f.sum()


@pytest.mark.parametrize("n,nb,nmax", [(31, 1, 64), (250, 3, 1000),
                                       (256, 2, 1024), (1000, 1, 8192),
                                       (5700, 1, 11400)])
def test_wake_and_csr(gpu_ctx, n, nb, nmax):
    a = space(gpu_ctx, n, density(n, nb, seed=7) if n < 5000
              else np.zeros((1, n, n), np.float32) + np.float32(1e-6))
    rng = np.random.default_rng(n)
    prof = (np.exp(-0.5 * np.linspace(-5, 5, n) ** 2)[None, :]
            * (1 + 0.1 * rng.random((nb, n)))).astype(np.float32)
    for b in range(nb):
        a.setProjection(0, b, prof[b])
    f = np.arange(nmax)
    z = (np.cbrt(f) * (0.87 + 0.5j)).astype(np.complex64)
    zi = V.Impedance(gpu_ctx, z, 1e12)
    spacing = (nmax - n) // max(nb - 1, 1)
    field = V.ElectricField(a, zi, list(range(nb)), spacing if nb > 1 else 0,
                            wakescaling=1.0)
    got = field.wakePotential()
    zz = z.astype(np.complex128)[:nmax // 2 + 1]
    zz[nmax // 2:] = 0
    pad = np.zeros(nmax)
    for b in range(nb):
        pad[b * spacing:b * spacing + n] += prof[b]
    w = np.fft.irfft(np.fft.rfft(pad) * zz, nmax)
    want = np.stack([w[b * spacing:b * spacing + n] for b in range(nb)])
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
    # the spectrum twice: the CTAs' counters start over
    for _ in range(2):
        field.updateCSR(0.0)
    spec, power = field.getCSRSpectrum(), field.getCSRPower()
    dq = 12.0 / (n - 1)
    ff = np.abs(np.fft.rfft(prof.astype(np.float64), nmax)) ** 2
    want = dq * dq * z.real[:nmax // 2 + 1].astype(np.float64) * ff
    assert (np.abs(spec[:, :nmax // 2 + 1] - want).max()
            <= 2e-5 * want.max())
    pw = want.sum(1) / dq / (nmax - 1)
    assert np.abs(power / pw - 1).max() <= 2e-5
