"""sed_solve_temperature on either side of the lines between its forms (a
thread, a warp or a CTA per zone): every zone's temperature is the root of
emission - e_abs, and many zones of few bins are not solved by whole CTAs."""
import time

import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.engine import Engine
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu
PI, C_L, H, K, SB = 3.14159, 2.99792458e10, 6.6260755e-27, 1.380658e-16, 5.6704e-5


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_zones,n_bins,packets", [
    (1, 2, 3000), (129, 31, 3000), (3, 32, 3000), (4143, 2, 800), (4144, 2, 800), (16577, 8, 100),  # thread or warp
    (5, 33, 3000), (295, 64, 3000), (297, 64, 3000), (2367, 512, 300), (2369, 512, 300), (2400, 513, 300)])  # warp or CTA
def test_temperature_is_the_root(sed_lib, precision, n_zones, n_bins, packets):
    w = workloads.lightbulb_grey(n_packets=packets, n_zones=n_zones, n_bins=n_bins, radiative_eq=1, seed=11)
    g = w.nu_grid()
    assert g.n == n_bins
    e = Engine(w, precision=precision)
    e.step(1.0)
    T, bad = e.solve_temperature()
    assert bad == 0
    kap = e.opacity()["abs"].reshape(n_zones, g.n)
    t = e.tallies(J=False)
    e_abs = t["e_abs"]
    nu, dnu = g.center(), g.width()

    def f(t):
        with np.errstate(over="ignore"):
            B = 2 * H * nu ** 3 / C_L ** 2 / np.expm1(H * nu / K / t[:, None])
        return (4 * PI * kap * B * dnu).sum(1) - e_abs

    lo, hi = np.full(n_zones, 1000.0), np.full(n_zones, 1e8)
    ok = (f(lo) < 0) & (f(hi) > 0)
    assert ok.mean() > 0.99
    for _ in range(100):
        m = 0.5 * (lo + hi)
        up = f(m) < 0
        lo, hi = np.where(up, m, lo), np.where(up, hi, m)
    # Brent ends within tol1 = 6e-8 T + 0.5e-2 K of the root, one step of at most that beyond
    assert np.all(np.abs(T - lo)[ok] <= (2e-2 + 2.5e-7 * lo)[ok])
    # set from the radiation energy density instead
    T, _ = e.solve_temperature(1)
    assert np.allclose(T, (t["e_rad"] / 7.5657e-15) ** 0.25, rtol=1e-4)
    e.close()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
def test_many_zones_of_one_bin_take_a_thread_each(sed_lib, precision):
    """64^3 zones of one bin: 0.5 ms with a thread per zone, 24 ms with a CTA
    (whose threads all repeat the root search); the line is at 5 ms."""
    w = grey_box(20000, shape=(64, 64, 64), seed=3)
    w.params["transport_nu_grid"] = [1e14, 1e16, 9.9e15, 1]
    e = Engine(w, precision=precision)
    assert e.nn == 1
    e.step(1.0)
    ms = []
    for _ in range(8):
        t0 = time.perf_counter()
        T, bad = e.solve_temperature()
        ms.append(1e3 * (time.perf_counter() - t0))
    assert bad == 0 and np.all(T >= 1000.0)
    assert min(ms) < 5.0
    e.close()
