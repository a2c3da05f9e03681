"""The work this framework is used for, as measurable cases.

Kinds of case:

``batch``   bunches of one mesh size stepped together (``BunchBatch.run``):
            one output interval of a running scan -- ``steps`` solver steps,
            then the densities, profiles and charges on the host (pinned
            buffers), and with ``csr`` the CSR power of every step.
            chain 0 is the solver loop (wake kick, RF kick, drift,
            Fokker-Planck), chain 1 the rotation scheme.
``uneven``  the same for one batch of mixed mesh sizes and interpolation
            orders.
``plain``   the one-map-per-call solver loop (``PlainSolver``) over one
            output interval, and the quantities a run records then
            (projections, moments, wake, CSR spectrum and power); any mesh
            size, one bunch or a beam of several.
``train``   one Adam step of the warm-start network on a minibatch.
``well``    the potential-well start of a batch.

Every input comes from the seed.  ``exact`` restates each path in 64-bit
torch.
"""
import math

import numpy as np
import torch

DEV = "cuda:0"
C = 2.99792458e8
SPT = 1000                       # steps per synchrotron period


def listed():
    return [
        # the smallest call: a single coarse bunch advanced a few steps
        # (interactive use, set-up scans): launches and latency
        dict(name="one_128", kind="batch", n=128, nb=1, chain=0, it=4,
             clamp=False, steps=8, spt=500, csr=False),
        # many coarse bunches, a ragged count (a quick wide current scan)
        dict(name="scan_64x777", kind="batch", n=64, nb=777, chain=0, it=4,
             clamp=False, steps=50, spt=1000, csr=False),
        # the benchmark's current scan over the reference's default output
        # interval
        dict(name="scan_256x256", kind="batch", n=256, nb=256, chain=0, it=4,
             clamp=False, steps=100, spt=1000, csr=False),
        # the bursting bunch: fine mesh, CSR power of every step
        dict(name="burst_512", kind="batch", n=512, nb=1, chain=0, it=4,
             clamp=False, steps=100, spt=4000, csr=True),
        # the benchmark's uneven batch (meshes 128..1024, orders 2..4)
        dict(name="uneven_96", kind="uneven", nb=96, steps=20, spt=2000,
             mix=4),
        # the current scan on the rotation chain
        dict(name="rotation_256x256", kind="batch", n=256, nb=256, chain=1,
             it=4, clamp=False, steps=20, spt=1000, csr=False),
        # the plain loop on the reference's default mesh
        dict(name="plain_256", kind="plain", n=256, nb=1, chain=0, it=4,
             clamp=False, steps=50, spt=1000, csr=True, pad=8.0),
        # the plain single bunch of the benchmark: clamped cubic rotation
        dict(name="plain_rotation_256", kind="plain", n=256, nb=1, chain=1,
             it=4, clamp=True, steps=50, spt=500, csr=False, pad=2.0),
        # a three-bunch beam on an odd mesh, quadratic interpolation
        dict(name="plain_beam_251", kind="plain", n=251, nb=3, chain=0, it=3,
             clamp=False, steps=20, spt=1000, csr=True, pad=8.0),
        # a mesh wider than the batch takes
        dict(name="plain_2048", kind="plain", n=2048, nb=1, chain=0, it=4,
             clamp=False, steps=4, spt=4000, csr=True, pad=4.0),
        # one training step of the warm-start network at its own mesh
        dict(name="train_256", kind="train", B=64, side=256),
        # the potential-well start of a scan
        dict(name="well_256x64", kind="well", n=256, nb=64, iters=200,
             spt=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["batch", "batch", "batch", "uneven", "plain", "plain",
                       "train", "well"])
    spt = rng.choice([500, 1000, 2000, 4000])
    if kind == "batch":
        n = rng.choice([64, 128, 256, 512, 1024])
        chain = rng.choice([0, 0, 1])
        steps = _log(rng, 1, 100)
        # at most the cells x steps of the largest listed case of the chain
        most = (256 * 65536 * 100 if chain == 0 else 256 * 65536 * 20) \
            // (n * n * steps)
        nb = _log(rng, 1, max(1, min(most, 256 * 65536 // (n * n))))
        it = rng.choice([2, 3, 4, 4])
        return dict(kind="batch", n=n, nb=nb, chain=chain, it=it,
                    clamp=chain == 1 and it == 4 and rng.random() < 0.5,
                    steps=steps, spt=spt,
                    csr=chain == 0 and rng.random() < 0.3)
    if kind == "uneven":
        return dict(kind="uneven", nb=_log(rng, 4, 96),
                    steps=_log(rng, 2, 20), spt=spt,
                    mix=rng.randrange(1, 1 << 20))
    if kind == "plain":
        n = _log(rng, 48, 2048)
        chain = rng.choice([0, 1])
        it = rng.choice([2, 3, 4, 4])
        return dict(kind="plain", n=n, nb=rng.choice([1, 1, 2, 3]),
                    chain=chain, it=it,
                    clamp=chain == 1 and it == 4 and rng.random() < 0.5,
                    steps=max(1, min(50, int(4 * 2048 ** 2 // n ** 2 // 3))),
                    spt=spt, csr=rng.random() < 0.5,
                    pad=rng.choice([4.0, 8.0]))
    if kind == "train":
        return dict(kind="train", B=_log(rng, 1, 64),
                    side=rng.choice([64, 96, 128, 200, 256]))
    return dict(kind="well", n=rng.choice([64, 128, 256]),
                nb=_log(rng, 1, 64), iters=_log(rng, 20, 200), spt=spt)


# ----------------------------------------------------------------- inputs
def lattice(n, spt):
    """Ring quantities of the default options, in plain arithmetic."""
    sE, E0, f_rev, H, V_RF, alpha0 = 4.7e-4, 1.3e9, 9e6, 50.0, 1e6, 4e-3
    R = C / (2 * math.pi * f_rev)
    V0 = 1.602e-19 * (E0 / 510998.9) ** 4 / (3 * 8.854187817e-12 * R)
    V_eff = math.sqrt(V_RF * V_RF - V0 * V0)
    fs = f_rev * math.sqrt(alpha0 * H * V_eff / (2 * math.pi * E0))
    dE = sE * E0
    bl = C * dE / H / f_rev ** 2 / V_eff * fs
    dt = 1.0 / (fs * spt)
    t_damp = E0 / V0 / f_rev
    I_norm = (17045.0 / 510998.9 * 2 * math.pi * (dE * fs / f_rev) ** 2
              / V_eff / H * (bl / R) ** (1.0 / 3.0))
    delta = 12.0 / (n - 1)
    return dict(n=n, angle=2 * math.pi / spt, e1=2.0 / (fs * t_damp * spt),
                I_norm=I_norm, bl=bl, delta=delta, f_rev=f_rev,
                # wake scaling per unit of S
                scale=I_norm * dt * C / bl / (delta * sE * E0))


def currents(count, rng):
    """Normalised currents of a scan: log-spaced 0.01..1.5, jittered."""
    s = np.geomspace(0.01, 1.5, count) if count > 1 else np.array([0.6])
    return s * np.exp(rng.uniform(-0.05, 0.05, size=count))


def impedance(nmax, n, f_rev, bl):
    """Free-space CSR impedance Z(n) ~ n^(1/3) as a table of nmax entries."""
    f = np.arange(nmax) / (nmax - 1) * (n * C / (12.0 * bl))
    z = 376.730313461 * math.gamma(2 / 3) / 3 ** (1 / 3) \
        * np.cbrt(f / f_rev) * complex(math.sqrt(3) / 2, 0.5)
    return z.astype(np.complex64)


def simpson(n):
    w = torch.full((n,), 2.0, dtype=torch.float64, device=DEV)
    w[1::2] = 4.0
    w[0] = w[-1] = 1.0
    return w * (12.0 / (n - 1) / 3.0)


def densities(n, count, seed, shares=None):
    """Bunches near equilibrium with their own position, widths and ripple,
    each normalised to its share; float32 [count][n][n] on the GPU."""
    r = np.random.default_rng([seed, n, count])
    par = torch.tensor(r.uniform(-1, 1, size=(count, 6)), device=DEV)
    x = torch.linspace(-6, 6, n, dtype=torch.float64, device=DEV)
    out = torch.empty(count, n, n, dtype=torch.float32, device=DEV)
    w = simpson(n)
    for b in range(0, count, 32):
        a = par[b:b + 32, :, None, None]
        q = (x[None, :, None] - 0.1 * a[:, 0]) / (1 + 0.05 * a[:, 1])
        p = (x[None, None, :] - 0.1 * a[:, 2]) / (1 + 0.05 * a[:, 3])
        d = torch.exp(-0.5 * (q * q + p * p))
        d = d * (1 + 0.05 * torch.sin(3 * q + 4 * a[:, 4])
                 * torch.cos(2 * p + 4 * a[:, 5]))
        tot = torch.einsum("bxy,x,y->b", d, w, w)
        if shares is not None:
            tot = tot / torch.tensor(shares[b:b + 32], device=DEV)
        out[b:b + 32] = (d / tot[:, None, None]).float()
    return out


def uneven_mix(case):
    """(n, order) of every bunch of an uneven batch."""
    r = np.random.default_rng(case["mix"])
    return [(int(n), int(it)) for n, it in
            zip(r.choice([128, 256, 512, 1024], size=case["nb"]),
                r.choice([2, 3, 4], size=case["nb"]))]


def bunches(case, seed):
    """Groups of bunches sharing mesh and order: [(n, order, positions in
    the batch, currents, densities)]."""
    r = np.random.default_rng([seed, 1])
    if case["kind"] == "uneven":
        mix = uneven_mix(case)
        S = r.uniform(0.1, 1.5, size=len(mix))
    else:
        mix = [(case["n"], case.get("it", 4))] * case["nb"]
        S = (r.uniform(0.02, 0.45, size=len(mix)) if case["kind"] == "well"
             else currents(len(mix), r))
    out = []
    for n, it in sorted(set(mix)):
        idx = [i for i, m in enumerate(mix) if m == (n, it)]
        out.append((n, it, idx, S[idx],
                    densities(n, len(idx), 16 * seed + it)))
    return out


def shares_of(nb):
    return [1.0] if nb == 1 else [(b + 1) / (nb * (nb + 1) / 2)
                                  for b in range(nb)]


def network(case, seed):
    """Weights, moments and a minibatch of the warm-start network in the
    middle of a training run."""
    B, npix = case["B"], case["side"] ** 2
    g = torch.Generator(device=DEV).manual_seed(seed)

    def rnd(*s):
        return torch.randn(*s, generator=g, device=DEV)
    shapes = dict(w1=(128, 3), b1=(128,), w2=(128, 128), b2=(128,),
                  w3=(32, 128), b3=(32,), wd=(32, npix), bd=(npix,))
    fan = dict(w1=3, w2=128, w3=128, wd=32)
    w = {k: rnd(*s) / math.sqrt(fan.get(k, 100)) for k, s in shapes.items()}
    # gradients scale like 1 / npix: the moments a run would have by now
    m = {k: rnd(*s) * 0.3 / npix for k, s in shapes.items()}
    v = {k: (rnd(*s).abs() + 0.5).square() / npix ** 2
         for k, s in shapes.items()}
    x = (torch.rand(B, 3, generator=g, device=DEV) * 2 - 1).cpu().numpy()
    return w, m, v, x, rnd(B, npix)


class View:
    """A library buffer as a tensor's source; keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(
            shape=shape, typestr="<f4", data=(ptr, False), version=2)


def prepare(case, seed):
    from inovesa_gb300 import params as P
    from inovesa_gb300 import vfps as V
    ctx = V.Context(0)
    kind = case["kind"]
    if kind == "train":
        from inovesa_gb300 import warmstart as W
        net = W.WarmStartNet(ctx, case["side"] ** 2, seed=0)
        w, m, v, x, t = network(case, seed)
        for k in net.names:
            net.w[k].copy_(w[k])
            net.m[k].copy_(m[k])
            net.v[k].copy_(v[k])
            if k in net.w16:
                net.w16[k].copy_(w[k])
        net.step_count = 500
        return dict(kind=kind, ctx=ctx, net=net, x=x, target=t)
    if kind == "plain":
        n, nb = case["n"], case["nb"]
        p = P.derive(GridSize=n, StepsPerTs=case["spt"], padding=case["pad"],
                     S_csr=0.5)
        L = lattice(n, case["spt"])
        z = V.Impedance(ctx, impedance(p["padded_bins"], n, L["f_rev"],
                                       L["bl"]), p["fmax"])
        sh = shares_of(nb)
        d = densities(n, nb, seed, sh).cpu().numpy()
        s = solver_of(ctx, p, case, z, sh, d)
        dens = torch.as_tensor(View((ctx, s), s.t1.devicePointer(),
                                    (nb, n, n)), device=DEV)
        return dict(kind=kind, ctx=ctx, solver=s, z=z, density=dens,
                    steps=case["steps"], csr=case["csr"])
    groups = bunches(case, seed)
    total = sum(len(g[2]) for g in groups)
    descs, parts, zs = [None] * total, [None] * total, {}
    chain, clamp = case.get("chain", 0), case.get("clamp", False)
    for n, it, idx, S, d in groups:
        p = P.derive(GridSize=n, StepsPerTs=case["spt"], padding=2.0,
                     S_csr=1.0)
        if n not in zs:
            zs[n] = (len(zs), V.Impedance(
                ctx, impedance(p["padded_bins"], n, p["f_rev"], p["bl"]),
                p["fmax"]))
        h = d.cpu().numpy()
        for k, i in enumerate(idx):
            descs[i] = P.fill_desc(V.BunchDesc(), p, chain,
                                   Ib=p["I_norm"] * float(S[k]),
                                   impedance=zs[n][0], it=it, clamp=clamp)
            parts[i] = h[k].ravel()
    zl = [z for _, z in sorted(zs.values(), key=lambda e: e[0])]
    b = V.BunchBatch(ctx, descs, zl)
    b.upload(np.concatenate(parts))
    if case.get("csr"):
        b.set_csr(zl, [0] * total, [p["fc"]] * total,
                  [C / p["bl"]] * total, every=1, capacity=case["steps"])

    def pinned(count):
        return torch.empty(count, dtype=torch.float32,
                           pin_memory=True).numpy()
    return dict(kind=kind, ctx=ctx, batch=b, z=zl,
                steps=case.get("steps", 0), iters=case.get("iters", 0),
                csr=case.get("csr", False), density=pinned(b.cells),
                profiles=pinned(b.rows), filling=pinned(total))


def solver_of(ctx, p, case, z, shares, data):
    from inovesa_gb300.solver import PlainSolver
    nb = case["nb"]
    return PlainSolver(ctx, p, chain=case["chain"], wake_impedance=z,
                       csr_impedance=z if case["csr"] else None,
                       it=case["it"], clamp=case["clamp"], data=data,
                       fillings=shares, buckets=list(range(nb)),
                       spacing=bucket_spacing(case["n"]))


def bucket_spacing(n):
    return n + n // 8


# -------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["target"])
        return dict(loss=loss, g=net.g, w=net.w)
    if kind == "plain":
        s = state["solver"]
        s.step(state["steps"], csr=state["csr"])
        ps = s.t1
        ps.updateYProjection()
        ps.variance(0)
        ps.variance(1)
        out = dict(density=state["density"], profile=ps.getProjection(0),
                   energy=ps.getProjection(1), length=ps.getBunchLength(),
                   spread=ps.getEnergySpread(),
                   wake=s.wake_field.getWakePotentials())
        if state["csr"]:
            out["spectrum"] = s.rdtn.getCSRSpectrum()
            out["power"] = s.rdtn.getCSRPower()
        return out
    b = state["batch"]
    if kind == "well":
        b.potential_well(state["iters"])
        b.run(None, 0, state["density"], state["profiles"], state["filling"])
    else:
        b.run(None, state["steps"], state["density"], state["profiles"],
              state["filling"])
    out = dict(density=state["density"], profiles=state["profiles"],
               filling=state["filling"])
    if state["csr"]:
        out["power"] = b.csr()[1]
    return out


def work(case):
    """Bytes: the state read once and written once (a pass may keep it on
    the chip in between).  Flops: per cell and step the kicks and the drift
    (one Lagrange sum of `it` taps each), the Fokker-Planck sum (4 taps)
    and the projection, or the rotation's it x it taps; per row the wake
    sum."""
    kind = case["kind"]
    if kind == "train":
        B, npix = case["B"], case["side"] ** 2
        params = 33 * npix + 128 * 3 + 128 * 128 + 32 * 128 + 288
        return dict(bytes=4 * B * npix + 28 * params,
                    flops=6 * B * 32 * npix + 12 * params)
    if kind == "uneven":
        mix, chain = uneven_mix(case), 0
    else:
        mix = [(case["n"], case.get("it", 4))] * case["nb"]
        chain = case.get("chain", 0)
    cells = sum(n * n for n, _ in mix)
    rows = sum(n * n for n, _ in mix)
    if kind == "well":
        # per pass and cell: the exponent (4), its exponential and the sum
        return dict(bytes=4 * cells, flops=8 * cells * case["iters"])
    per = sum(n * n * (2 * (it * it + it + it + 4 + 1) + 40 if chain
                       else 2 * (3 * it + 4 + 1)) for n, it in mix)
    return dict(bytes=8 * cells, flops=case["steps"] * (per + 2 * rows))


# ------------------------------------------------------------------ exact
def lagrange(f, it):
    if it == 2:
        return [1 - f, f]
    if it == 3:
        return [f * (f - 1) / 2, 1 - f * f, f * (f + 1) / 2]
    return [-(f - 1) * (f - 2) * f / 6, (f + 1) * (f - 1) * (f - 2) / 2,
            (2 - f) * f * (f + 1) / 2, f * (f + 1) * (f - 1) / 6]


def kick(d, off, it, axis):
    """KickMap along y (off [bunch][x]) or x (off [y])."""
    nb, n, _ = d.shape
    pos = n // 2 + off
    base = torch.trunc(pos)
    f = pos - base
    first = base.long() - (it - 1) // 2
    c = lagrange(f, it)
    out = torch.zeros_like(d)
    i = torch.arange(n, device=d.device)
    for j in range(it):
        ok = (first + j >= 0) & (first + j < n) & (base >= 0)
        w = torch.where(ok, c[j], torch.zeros_like(f))
        if axis == 1:
            src = i[None, None, :] + (first + j - n // 2)[:, :, None]
            v = torch.gather(d, 2, src.clamp(0, n - 1))
            v = torch.where((src >= 0) & (src < n), v, 0.0)
            out += v * w[:, :, None]
        else:
            src = i[:, None] + (first + j - n // 2)[None, :]
            v = torch.gather(d, 1, src.clamp(0, n - 1).expand(nb, n, n))
            v = torch.where((src >= 0) & (src < n), v, 0.0)
            out += v * w[None, None, :]
    return out


class Rotation:
    def __init__(self, n, angle, it, clamp):
        a = torch.linspace(-6, 6, n, dtype=torch.float64, device=DEV)
        cs, sn, dl = math.cos(-angle), math.sin(-angle), 12.0 / (n - 1)
        zb = (n - 1) / 2
        x = (cs * a[:, None] - sn * a[None, :]) / dl + zb
        y = (sn * a[:, None] + cs * a[None, :]) / dl + zb
        x1, y1 = torch.trunc(x), torch.trunc(y)
        self.ok = (x1 >= 0) & (x1 < n) & (y1 >= 0) & (y1 < n)
        self.cx, self.cy = lagrange(x - x1, it), lagrange(y - y1, it)
        self.x, self.y = x1.long(), y1.long()
        self.n, self.it, self.clamp = n, it, clamp

    def __call__(self, d):
        n, it, h = self.n, self.it, (self.it - 1) // 2
        flat = d.reshape(len(d), -1)
        out = torch.zeros_like(d)
        lo = torch.full_like(d, math.inf) if self.clamp else None
        hi = torch.zeros_like(d) if self.clamp else None
        for i in range(it):
            for j in range(it):
                xs, ys = self.x + i - h, self.y + j - h
                ok = (self.ok & (xs >= 0) & (xs < n) & (ys >= 0) & (ys < n))
                at = torch.where(ok, xs * n + ys, 0)
                v = flat[:, at.reshape(-1)].reshape(d.shape)
                out += v * torch.where(ok, self.cx[i] * self.cy[j], 0.0)
                if self.clamp and i in (1, 2) and j in (1, 2):
                    hi, lo = torch.maximum(hi, v), torch.minimum(lo, v)
        if self.clamp:
            out = torch.maximum(torch.minimum(out, hi), lo)
        return out


def fokker_planck(n, e1):
    """Weights [5][n] of the offsets -2..2 (damping and diffusion, cubic
    derivative)."""
    dl = 12.0 / (n - 1)
    p = np.linspace(-6, 6, n)
    w = np.zeros((5, n))
    for j in range(2, n - 2):
        d = e1 / (6 * dl) * p[j]
        if j < int((n - 1) / 2):
            w[:, j] = [d, -6 * d, 1 + e1 + 3 * d, 2 * d, 0]
        else:
            w[:, j] = [0, -2 * d, 1 + e1 - 3 * d, 6 * d, -d]
        w[1:4, j] += np.array([1, -2, 1]) * e1 / dl ** 2
    return torch.tensor(w, device=DEV)


class Loop:
    """The solver step of bunches on one mesh, in 64 bits."""

    def __init__(self, n, it, chain, clamp, spt, z, scale, pos):
        L = lattice(n, spt)
        self.n, self.it, self.chain, self.L = n, it, chain, L
        self.ws, self.z, self.pos = simpson(n), z, pos
        self.scale = scale            # [bunch], wake scaling
        x = torch.arange(n, dtype=torch.float64, device=DEV)
        self.rf = math.tan(L["angle"]) * ((n - 1) / 2 - x)
        self.dr = L["angle"] * (x * L["delta"] - 6) / L["delta"]
        self.fp = fokker_planck(n, L["e1"])
        self.rot = Rotation(n, L["angle"], it, clamp) if chain else None

    def profile(self, d):
        return d @ self.ws

    def wake(self, P):
        """Every bunch's wake from the padded profile: of all bunches at
        their positions, or (pos None) of each bunch alone."""
        nmax, nb = len(self.z), len(P)
        pad = torch.zeros(nb, nmax, dtype=torch.float64, device=DEV)
        if self.pos is None:
            pad[:, :self.n] = P
        else:
            for b, at in enumerate(self.pos):
                pad[:, at:at + self.n] += P[b]
        zz = self.z[:nmax // 2 + 1].clone()
        zz[nmax // 2:] = 0
        w = torch.fft.irfft(torch.fft.rfft(pad) * zz, n=nmax)
        if self.pos is None:
            w = w[:, :self.n]
        else:
            w = torch.stack([w[b, at:at + self.n]
                             for b, at in enumerate(self.pos)])
        return w * self.scale[:, None]

    def step(self, d, W):
        nb = len(d)
        if self.chain == 0:
            d = kick(d, W, self.it, 1)
            d = kick(d, self.rf.expand(nb, -1), self.it, 1)
            d = kick(d, self.dr, self.it, 0)
        else:
            d = kick(self.rot(d), W, self.it, 1)
        out = torch.zeros_like(d)
        n = self.n
        for o in range(5):
            out[:, :, 2:n - 2] += self.fp[o, 2:n - 2] * d[:, :, o:n - 4 + o]
        return out

    def spectrum(self, P, fc=23e9):
        nmax, dl = len(self.z), self.L["delta"]
        k = torch.arange(nmax // 2 + 1, dtype=torch.float64, device=DEV)
        df = 1 / dl / (nmax - 1)
        cut = 1 - torch.exp(-(C / self.L["bl"] * df * k / fc) ** 2)
        ff = torch.fft.rfft(P, n=nmax)
        s = torch.zeros(len(P), nmax, dtype=torch.float64, device=DEV)
        s[:, :nmax // 2 + 1] = (dl * dl * cut * self.z.real[:nmax // 2 + 1]
                                * ff.abs() ** 2)
        return s, s.sum(1) * df


def exact_loop(case, n, it, S, nmax, pos):
    L = lattice(n, case["spt"])
    z = torch.tensor(impedance(nmax, n, L["f_rev"], L["bl"])
                     .astype(np.complex128), device=DEV)
    sc = torch.tensor(np.asarray(S), dtype=torch.float64, device=DEV) \
        * L["scale"]
    return Loop(n, it, case.get("chain", 0), case.get("clamp", False),
                case["spt"], z, sc, pos)


def exact_batch(case, seed):
    groups = bunches(case, seed)
    total = sum(len(g[2]) for g in groups)
    dens, prof = [None] * total, [None] * total
    fill, power = np.zeros(total), []
    for n, it, idx, S, d0 in groups:
        for at in range(0, len(idx), 32):
            part = idx[at:at + 32]
            M = exact_loop(case, n, it, S[at:at + 32], 2 * n, None)
            d = d0[at:at + 32].double()
            pw = []
            for _ in range(case["steps"]):
                P = M.profile(d)
                if case.get("csr"):
                    pw.append(M.spectrum(P)[1])
                d = M.step(d, M.wake(P))
            f = P @ M.ws
            P = M.profile(d)
            for k, i in enumerate(part):
                dens[i] = d[k].cpu().numpy().ravel()
                prof[i] = P[k].cpu().numpy()
                fill[i] = float(f[k])
            if pw:
                power.append(torch.stack(pw).cpu().numpy())
    out = dict(density=np.concatenate(dens), profiles=np.concatenate(prof),
               filling=fill)
    if power:
        out["power"] = np.concatenate(power, axis=1)
    return out


def exact_plain(case, seed):
    n, nb = case["n"], case["nb"]
    sh = shares_of(nb)
    nmax = 1 << (int(math.ceil(n * case["pad"])) - 1).bit_length()
    pos = [b * bucket_spacing(n) for b in range(nb)]
    M = exact_loop(case, n, case["it"], [0.5] * nb, nmax, pos)
    d = densities(n, nb, seed, sh).double()
    for _ in range(case["steps"]):
        P = M.profile(d)
        W = M.wake(P)
        if case["csr"]:
            spec, power = M.spectrum(P)
        d = M.step(d, W)
    fill = P @ M.ws
    P = M.profile(d)
    E = torch.einsum("bxy,x->by", d, M.ws)
    a = torch.linspace(-6, 6, n, dtype=torch.float64, device=DEV)

    def rms(pr):
        k = M.L["delta"] / fill
        av = (pr @ a) * k
        return ((pr * (a - av[:, None]) ** 2).sum(1) * k).sqrt()
    out = dict(density=d, profile=P, energy=E, length=rms(P), spread=rms(E),
               wake=W)
    if case["csr"]:
        out.update(spectrum=spec, power=power)
    return {k: v.cpu().numpy() for k, v in out.items()}


def exact_train(case, seed):
    w, m, v, x, t = network(case, seed)
    u = {k: (a.bfloat16() if k.startswith("w") else a).double()
         for k, a in w.items()}
    x, t = torch.tensor(x, device=DEV).double(), t.double()
    h1 = torch.tanh(x @ u["w1"].T + u["b1"])
    h2 = torch.tanh(h1 @ u["w2"].T + u["b2"])
    zz = h2 @ u["w3"].T + u["b3"]
    e = zz @ u["wd"] + u["bd"] - t
    g = {}
    dy = 2 * e / e.numel()
    g["wd"], g["bd"] = zz.T @ dy, dy.sum(0)
    dz = dy @ u["wd"].T
    g["w3"], g["b3"] = dz.T @ h2, dz.sum(0)
    d2 = (dz @ u["w3"]) * (1 - h2 * h2)
    g["w2"], g["b2"] = d2.T @ h1, d2.sum(0)
    d1 = (d2 @ u["w2"]) * (1 - h1 * h1)
    g["w1"], g["b1"] = d1.T @ x, d1.sum(0)
    new = {}
    for k, a in g.items():
        mm = 0.9 * m[k].double() + 0.1 * a
        vv = 0.999 * v[k].double() + 0.001 * a * a
        new[k] = w[k].double() - 1e-3 * (mm / (1 - 0.9 ** 501)) / (
            (vv / (1 - 0.999 ** 501)).sqrt() + 1e-8)
    return dict(loss=float((e * e).mean()),
                g={k: a.cpu().numpy() for k, a in g.items()},
                w={k: a.cpu().numpy() for k, a in new.items()})


def exact_well(case, seed):
    (n, it, idx, S, _), = bunches(case, seed)
    dens, prof, fill = [], [], []
    for at in range(0, len(idx), 32):
        M = exact_loop(case, n, it, S[at:at + 32], 2 * n, None)
        nb, dl = len(idx[at:at + 32]), M.L["delta"]
        T = M.L["angle"] / dl ** 2

        def integral(f):
            out = torch.zeros_like(f)
            out[..., 1:] = torch.cumsum((f[..., 1:] + f[..., :-1]) / 2, -1)
            return out
        G = integral(M.dr)
        G = G - G.min()
        W = torch.zeros(nb, n, dtype=torch.float64, device=DEV)
        P = None
        for k in range(case["iters"] + 1):
            F = -(M.rf + W)
            ex = -(integral(F)[:, :, None] + G
                   + 0.5 * F[:, :, None] * M.dr) / T
            d = torch.exp(ex - ex.amax((1, 2), keepdim=True))
            d = d / torch.einsum("bxy,x,y->b", d, M.ws, M.ws)[:, None, None]
            r = M.profile(d)
            P = r if P is None else P + 0.5 * (r - P)
            W = M.wake(P)
        dens.append(d.reshape(nb, -1).cpu().numpy())
        prof.append(r.cpu().numpy())
        fill.append((r @ M.ws).cpu().numpy())
    return dict(density=np.concatenate(dens).ravel(),
                profiles=np.concatenate(prof).ravel(),
                filling=np.concatenate(fill))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return exact_train(case, seed)
    if kind == "plain":
        return exact_plain(case, seed)
    if kind == "well":
        return exact_well(case, seed)
    return exact_batch(case, seed)
