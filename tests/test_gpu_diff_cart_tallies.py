"""Zone tallies of the weighted forward on 3D grids, with FP32 tables (in copies
up to 8192 cells, added up directly beyond) and in FP64: means over independent
steps agree."""
import numpy as np
import pytest

from pubsed_b200 import abi
from pubsed_b200.adjoint import DiffEngine
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 2), (16, 16, 32), (16, 16, 33)])
def test_tallies_of_both_precisions_agree(sed_lib, shape):
    steps = 12
    got = []
    for precision in (abi.PREC_FP64, abi.PREC_MIXED):
        w = grey_box(3000, shape=shape, seed=17, radiative_eq=0)
        w.params["opacity_epsilon"] = 0.05
        e = DiffEngine(w, n_bands=4, precision=precision)
        e.tables()
        rows = []
        for s in range(steps):
            e.forward(np.ones((e.nz, 4)), step=s + 100 * (precision == abi.PREC_MIXED))
            t = e.tallies(J=False)
            half = np.arange(e.nz) < (e.nz + 1) // 2
            v = w.zones.vol
            rows.append([(v * t["e_abs"])[half].sum(), (v * t["e_abs"]).sum(), (v * t["fr"]).sum(), (v * t["e_rad"]).sum()])
        got.append(np.array(rows))
        e.close()
    a, b = got
    assert np.all(a[:, :2] > 0) and np.all(b[:, :2] > 0)
    # six standard errors of the difference of two means over 12 independent steps
    err = np.sqrt((a.var(0, ddof=1) + b.var(0, ddof=1)) / steps)
    assert np.all(np.abs(a.mean(0) - b.mean(0)) <= 6 * err), (a.mean(0), b.mean(0), err)
