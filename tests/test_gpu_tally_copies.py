"""The mean intensity tallied in copies (few addresses) against the same
histories tallied bin by bin in one array."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


def _run(sed_lib, w, precision):
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    g.set_opacity(1.0)
    st = g.transport(1.0)
    out = (st["n_segments"], g.spectrum()[1], g.tallies())
    g.close()
    return out


# zones x bins lies above the copies' limit (65536 values) for the run that
# stores J per bin; without bins there are 32 copies (up to 2048 zones), 31, 2
# and none
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_zones,n_bins", [(1, 65537), (7, 9363), (2048, 33), (2049, 33), (32768, 3), (32769, 3)])
def test_mean_intensity_copies(sed_lib, n_zones, n_bins, precision):
    def model(store):
        w = workloads.lightbulb_grey(n_packets=3000, n_zones=n_zones, n_bins=n_bins, seed=21)
        w.params["transport_store_Jnu"] = store
        return w
    seg1, click1, t1 = _run(sed_lib, model(1), precision)
    seg0, click0, t0 = _run(sed_lib, model(0), precision)
    assert seg1 == seg0 and np.array_equal(click1, click0)
    # e_rad is the zone's sum either way: at most seg1 terms of one sign, each
    # scaled and summed with a few roundings
    np.testing.assert_allclose(t0["e_rad"], t1["e_rad"], rtol=(seg1 + 64) * 2.0**-52, atol=0)


# 210 cells x 314 bins lie above the limit, 210 cells take 32 copies
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
def test_mean_intensity_copies_3d(sed_lib, precision):
    runs = []
    for store in (1, 0):
        w = grey_box(2000, shape=(6, 5, 7), seed=8, radiative_eq=1)
        d = workloads.log_delta_for_bins(1e14, 1e16, 314)
        w.params["transport_nu_grid"] = [1e14, 1e16, d, 1]
        w.params["transport_store_Jnu"] = store
        runs.append(_run(sed_lib, w, precision))
    (seg1, click1, t1), (seg0, click0, t0) = runs
    assert seg1 == seg0 and np.array_equal(click1, click0)
    np.testing.assert_allclose(t0["e_rad"], t1["e_rad"], rtol=(seg1 + 64) * 2.0**-52, atol=0)
