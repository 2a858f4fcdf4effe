"""Loaded emissivity CDFs that end below 1: a deviate past a row's end takes the
last bin in every form of the packet kernel."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("kind", ["sphere", "static sphere", "box"])
@pytest.mark.parametrize("end", [0.0, 0.7])
def test_deviates_past_the_end_take_the_last_bin(sed_lib, precision, kind, end):
    n = 2000
    if kind == "box":
        w = grey_box(n, shape=(5, 6, 4), seed=3, radiative_eq=1)
    else:
        w = workloads.lightbulb_grey(n_packets=n, n_zones=9, n_bins=64, radiative_eq=1, seed=3)
        if kind == "static sphere":
            w.zones.homologous = 0
            w.zones.v = np.zeros(9)
    e = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    e.set_opacity(1.0)
    t = e.opacity()
    g = w.nu_grid()
    e.load_opacity(t["abs"], t["scat"], end * t["emis_cdf"], t["eps_imc"])
    e.record(True)
    st = e.transport(1.0)
    assert st["n_escaped"] + st["n_absorbed"] + st["n_stopped"] == n
    r = e.records(n)
    nu = r["state"][:, 8]
    beta = 0.0 if kind == "static sphere" else 0.06  # two transforms, at up to 1.7e9 cm/s in a box's corner
    assert np.all((nu >= g.min * (1 - 2 * beta)) & (nu <= g.right[-1] * (1 + 2 * beta)))
    # without the first bins' share the last bin holds most of what was re-emitted
    last = (nu >= g.right[-2] * (1 - 2 * beta)) & (r["fate"] == 2)
    assert np.count_nonzero(last) > n // 20
    e.close()
