"""The packed bins of the 1D mixed packet kernel: packets on them, on the
separate tables (a context that has no packed bins), and on tables written by
something else than an opacity build have the same histories to the bit."""
import copy
import ctypes as C

import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.grids import LocGrid
import oracle_lib

pytestmark = pytest.mark.gpu
N = 2000


def _records(e):
    e.record(True)
    e.lib.sed_set_rng_step(e.ctx, 0)
    e.transport(1.0)
    return e.records(N)


def _same(a, b):
    for k in ("fate", "ind", "draws", "state"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n_bins,radiative_eq", [(2, 1), (40, 0), (700, 1)])
def test_packed_and_separate_tables_agree(sed_lib, n_bins, radiative_eq):
    w = workloads.type_ia(n_packets=N, n_zones=27, n_lines=4000, n_bins=n_bins, spectrum_bins=32, seed=9,
                          radiative_eq=radiative_eq)
    a = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    a.set_opacity(1.0)
    # a context whose tables were sized for a 3D grid of as many zones holds no packed bins
    z = copy.copy(w.zones)
    z.type = abi.GRID_3D_CART
    edge = float(z.r_out[-1])
    ax = LocGrid(np.array([-edge / 3, edge / 3, edge]), -edge, 0.0, abi.LOC_FLEX)
    z.axes, z.shape = [ax, ax, ax], (3, 3, 3)
    w3 = copy.copy(w)
    w3.zones = z
    b = oracle_lib.Engine(sed_lib, "sed_", w3, precision=abi.PREC_MIXED)
    b.w = w
    b.set_grid()
    b.set_opacity(1.0)
    _same(_records(a), _records(b))
    a.close()
    b.close()


def test_scaled_and_restored_tables(sed_lib):
    """sed_diff_scale_extinction rewrites the {abs, scat} tables: a plain step
    then runs on the scaled ones, and on the built ones once they are back."""
    w = workloads.type_ia(n_packets=N, n_zones=12, n_lines=3000, n_bins=200, spectrum_bins=32, seed=10)
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    g.set_opacity(1.0)
    built, t = _records(g), g.opacity()
    r = np.linspace(0.5, 2.0, 12)
    P = r.ctypes.data_as(abi._dp)
    assert sed_lib.sed_diff_scale_extinction(g.ctx, P) == 0
    scaled = _records(g)
    assert not np.array_equal(scaled["draws"], built["draws"])
    f = np.repeat(r, 200)
    s = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    s.load_opacity(t["abs"] * f, t["scat"] * f, t["emis_cdf"], t["eps_imc"])
    _same(scaled, _records(s))
    assert sed_lib.sed_diff_scale_extinction(g.ctx, C.cast(None, abi._dp)) == 0
    _same(built, _records(g))
    g.close()
    s.close()
