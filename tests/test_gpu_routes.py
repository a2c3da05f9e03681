"""The kernels that keep densities on the chip (k_bres, k_bcol), where calls
are known to take them (vfps_batch_route), against the per-step kernels:
several bunches per cluster, halos of several rows, CSR powers.

Tolerances as in test_gpu_resident.py."""
import pytest

import test_gpu_resident as R

pytestmark = pytest.mark.gpu


def sides(ctx, monkeypatch, steps, rounds, csr=False, **kw):
    """test_gpu_resident.both, with the first side's calls on the chip and
    the second's not."""
    probe, _, _ = R.batch(ctx, **kw)
    for k in steps:
        route = probe.route(k)
        assert route["resident"] and route["rounds"] == rounds, (k, route)
    monkeypatch.setenv("VFPS_RING_KERNEL", "steps")
    probe, _, _ = R.batch(ctx, **kw)
    assert not probe.route(1000)["resident"]
    monkeypatch.delenv("VFPS_RING_KERNEL")
    a, b = R.both(ctx, monkeypatch, steps, csr=csr, **kw)
    R.check(a, b)


def two_rounds_512(ctx):
    """Bunches that k_bcol takes in two rounds: twice the clusters that run at
    a time (seven on most devices)."""
    for nb in (14, 16, 12, 18, 20):
        b, _, _ = R.batch(ctx, n=512, nb=nb, spt=4000)
        route = b.route(6)
        if route["resident"] and route["rounds"] == 2:
            return nb
    raise AssertionError("no batch of two rounds")


# k_bcol: seven clusters at a time, so 14 bunches are two rounds; odd and even
# numbers of steps (the buffers and barriers of the second bunch carry on
# where the first ended); 4000 steps a period: the drift reads two rows on
# either side at most
@pytest.mark.parametrize("steps", [(11, 6), (12,), (7, 7)])
@pytest.mark.parametrize("csr", [False, True])
def test_second_round_512(gpu_ctx, monkeypatch, steps, csr):
    sides(gpu_ctx, monkeypatch, steps, 2, csr=csr, n=512,
          nb=two_rounds_512(gpu_ctx), spt=4000)


@pytest.mark.parametrize("n,nb,more", [(512, 1, False), (256, 100, True),
                                       (64, 700, True)])
def test_rounds_and_csr(gpu_ctx, monkeypatch, n, nb, more):
    b, _, _ = R.batch(gpu_ctx, n=n, nb=nb, spt=4000)
    route = b.route(11)
    assert route["resident"] and (route["rounds"] >= 2) == more
    sides(gpu_ctx, monkeypatch, (11, 12), route["rounds"], csr=True, n=n,
          nb=nb, spt=4000)


# the power that k_bcol records, in one round and two, against 64 bits
@pytest.mark.parametrize("rounds", [1, 2])
def test_csr_power_512(gpu_ctx, monkeypatch, rounds):
    nb = 1 if rounds == 1 else two_rounds_512(gpu_ctx)
    make = R.batch

    def batch(ctx, n, count):
        b, p, z = make(ctx, n, count, spt=4000)
        assert b.route(12)["resident"]
        return b, p, z
    monkeypatch.setattr(R, "batch", batch)
    R.test_csr_power(gpu_ctx, 512, nb)


# 201 steps a period: the drift's shift changes every 32 columns, so the
# lattices are regular, with up to 2 and 4 rows of drift
@pytest.mark.parametrize("n,nb", [(128, 2), (128, 30), (256, 2), (256, 30)])
@pytest.mark.parametrize("it", [2, 4])
def test_wide_drift(gpu_ctx, monkeypatch, n, nb, it):
    b, _, _ = R.batch(gpu_ctx, n=n, nb=nb, it=it, spt=201)
    assert b.kernel_tiles()["k_bmaps0f"] > 0
    sides(gpu_ctx, monkeypatch, (6, 7), b.route(6)["rounds"], csr=True, n=n,
          nb=nb, it=it, spt=201)


def test_launches_stay_short(gpu_ctx):
    """A launch of many steps takes about a second at most: a step of 256-row
    bunches is 4.2 us a round of clusters at most, and 4096 bunches are more
    than a hundred rounds.  A call of more steps is several launches."""
    p = R.P.derive(GridSize=256, StepsPerTs=1000, padding=2.0, S_csr=1.0)
    z = R.V.makeImpedance(gpu_ctx, **R.P.wake_impedance_args(p))
    d = R.P.fill_desc(R.V.BunchDesc(), p, 0, Ib=p["I_norm"], impedance=0)
    b = R.V.BunchBatch(gpu_ctx, [d] * 4096, [z])
    route = b.route(100000)
    assert route["resident"] and route["rounds"] > 100
    assert 1000 <= route["launch_steps"] <= 1e6 / 4.2 / route["rounds"]
    small, _, _ = R.batch(gpu_ctx, n=64, nb=2)
    most = small.route(100000)["launch_steps"]
    assert most == 8192
    small.step(most + 3)
    assert gpu_ctx.device_status() == 0


def test_routes(gpu_ctx):
    b, _, _ = R.batch(gpu_ctx, n=128, nb=3)
    assert b.route(100) == dict(b.route(100), resident=True, rounds=1)
    assert not b.route(0)["resident"]
    b.set_wake_mode(1)
    assert b.route(100) == dict(resident=False, rounds=0, launch_steps=1)
    b.set_wake_mode(0)
    assert b.route(100)["resident"]
    b, _, _ = R.batch(gpu_ctx, n=128, nb=3, wake=False)
    assert b.route(100)["resident"]
    b.set_beams([1, 1, 0], [0, 1, 0], 160)
    assert not b.route(100)["resident"]
    wide, _, _ = R.batch(gpu_ctx, n=1024, nb=1, spt=4000)
    assert not wide.route(100)["resident"]
    assert gpu_ctx.device_status() == 0
