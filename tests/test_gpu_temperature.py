"""sed_solve_temperature at the sizes where its CTA per zone can go wrong: one
bin, fewer bins than threads, bins that are no multiple of the CTA, the
largest row kept in shared memory and rows beyond it, one zone; both forms.
Each zone's temperature is the root of emission - e_abs found by bisection in
numpy from the tables and tallies the library returns."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.engine import Engine

pytestmark = pytest.mark.gpu
PI, C_L, H, K, SB = 3.14159, 2.99792458e10, 6.6260755e-27, 1.380658e-16, 5.6704e-5


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_zones,n_bins", [(1, 64), (33, 1), (5, 255), (7, 257), (3, 6144), (3, 6145)])
def test_temperature_is_the_root(sed_lib, precision, n_zones, n_bins):
    w = workloads.lightbulb_grey(n_packets=4000, n_zones=n_zones, n_bins=n_bins, radiative_eq=1, seed=11)
    g = w.nu_grid()
    assert (g.n == 1) if n_bins == 1 else (g.n >= n_bins - 1)
    e = Engine(w, precision=precision)
    e.step(1.0)
    T, bad = e.solve_temperature()
    assert bad == 0
    kap = e.opacity()["abs"].reshape(n_zones, g.n)
    e_abs = e.tallies(J=False)["e_abs"]
    nu, dnu = g.center(), g.width()

    def f(t):
        if g.n == 1:
            return 4 * PI * kap[:, 0] * SB / PI * t ** 4 - e_abs
        with np.errstate(over="ignore"):
            B = 2 * H * nu ** 3 / C_L ** 2 / np.expm1(H * nu / K / t[:, None])
        return (4 * PI * kap * B * dnu).sum(1) - e_abs

    lo, hi = np.full(n_zones, 1000.0), np.full(n_zones, 1e8)
    assert np.all(f(lo) < 0) and np.all(f(hi) > 0)
    for _ in range(100):
        m = 0.5 * (lo + hi)
        up = f(m) < 0
        lo, hi = np.where(up, m, lo), np.where(up, hi, m)
    # Brent ends within tol1 = 6e-8 T + 0.5e-2 K of the root, one step of at most that beyond
    assert np.all(np.abs(T - lo) <= 2e-2 + 2.5e-7 * lo)
    e.close()
