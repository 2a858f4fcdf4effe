"""The spectra of the 3D mixed packet kernel, packet by packet: every escaped
packet is counted once, in the bin its recorded end state belongs to, whether
the kernel leaves it in its emission slot for the binning kernel or counts it
itself; and the escaped energy agrees with the oracle's."""
import numpy as np
import pytest

from pubsed_b200 import abi
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


def _bin(g, x):
    """locate_array::locate on a grid's walls: below the grid 0, above it n."""
    if g.n == 1:
        return np.zeros(x.size, int)
    return np.where(x < g.min, 0, np.searchsorted(g.right, x, side="right"))


def _spectrum(w, r):
    """{flux, click} of recorded packets by spectrum_array::count's rules."""
    tg, ng, mg, pg = w.spectrum_grids()
    s = r["state"][r["fate"] == 2]
    phi = np.arctan2(s[:, 4], s[:, 3])
    phi = np.where(phi < 0, phi + 2 * 3.14159, phi)
    t, l, m, p = _bin(tg, s[:, 6]), _bin(ng, s[:, 8]), _bin(mg, s[:, 5]), _bin(pg, phi)
    l = np.where(l >= ng.n, 0, l)
    ok = (t < tg.n) & (m < mg.n) & (p < pg.n)
    i = ((t * ng.n + l) * mg.n + m) * pg.n + p
    size = tg.n * ng.n * mg.n * pg.n
    return np.bincount(i[ok], s[ok, 7], size), np.bincount(i[ok], minlength=size).astype(float)


def _agree(w, e, n):
    r = e.records(n)
    flux, click = e.spectrum()
    f, c = _spectrum(w, r)
    assert np.array_equal(click, c)
    assert np.allclose(flux, f, rtol=1e-12, atol=0)
    return r


@pytest.mark.parametrize("n,shape,radiative_eq", [(1, (1, 1, 1), 1), (3000, (4, 1, 7), 0), (40_000, (5, 6, 4), 1)])
def test_escaped_packets_are_counted_where_they_belong(sed_lib, n, shape, radiative_eq):
    w = grey_box(n, shape=shape, seed=8, radiative_eq=radiative_eq)
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    for e in (o, g):
        e.set_opacity(1.0)
        e.record(True)
        e.transport(1.0)
    rg, ro = _agree(w, g, n), o.records(n)
    # escaped energies: independent runs of n packets, each sum with variance n <e^2>
    eg, eo = (np.where(r["fate"] == 2, r["state"][:, 7], 0.0) for r in (rg, ro))
    if n > 100:
        assert abs(eg.sum() - eo.sum()) <= 5 * np.sqrt(n * (eg.var() + eo.var()))
    o.close()
    g.close()


def test_packets_beside_a_census_are_counted_where_they_belong(sed_lib):
    """A carried packet makes the kernel emit and count the packets itself."""
    n = 4000
    w = grey_box(n, shape=(5, 4, 6), seed=8, radiative_eq=1)
    w.params["transport_steady_iterate"] = 0
    e = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    erad = np.ones(e.nz)
    assert sed_lib.sed_initialize_particles(e.ctx, 1, erad.ctypes.data_as(abi._dp)) == 0
    dt = 40 * 86400.0  # longer than any packet stays
    e.set_opacity(dt)
    e.record(True)
    e.transport(dt)
    r = _agree(w, e, n + 1)
    assert np.count_nonzero(r["fate"] == 2) > n // 2
    e.close()
