"""How far the potential-well states are from 64 bits (perf/cases.py's
restatement on the same inputs).

The bounds are what one FP32 thread block per bunch with the sums in sequence
reaches, with 15 % on top: root mean square relative to the states' own,
densities 8.3e-7 and profiles 4.8e-7 on 256 rows, 6.6e-7 and 4.6e-7 on 128,
1.05e-6 and 5.6e-7 on 64.  (The exponent of a tail cell is about 40, its
rounding 40 eps / 2 = 2.4e-6 of the cell.)"""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb,iters,spt,dens,prof", [
    (256, 7, 30, 500, 8.3e-7, 4.8e-7),
    (128, 5, 40, 1000, 6.6e-7, 4.6e-7),
    (64, 5, 40, 2000, 1.05e-6, 5.6e-7),
])
def test_error_against_64_bits(n, nb, iters, spt, dens, prof):
    case = dict(kind="well", n=n, nb=nb, iters=iters, spt=spt)
    err = {"density": [], "profiles": []}
    for seed in (1, 2, 3, 4):
        got = cases.run(cases.prepare(case, seed))
        want = cases.exact(case, seed)
        for k, e in err.items():
            w = np.asarray(want[k], np.float64).ravel()
            d = np.asarray(got[k], np.float64).ravel() - w
            e.append(np.sqrt((d * d).mean() / (w * w).mean()))
    assert np.mean(err["density"]) <= 1.15 * dens, err
    assert np.mean(err["profiles"]) <= 1.15 * prof, err
