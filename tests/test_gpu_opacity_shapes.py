"""The opacity build against the oracle at the sizes where its split over the
chip can go wrong: fewer bins than the warps of a CTA, bins that are no
multiple of it, one zone, a zone more than a tile, many zones with few bins;
both forms, with the tolerances of test_gpu_opacity.py."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib

pytestmark = pytest.mark.gpu


def _maxrel(a, b):
    s = np.abs(b)
    s = np.where(s == 0, 1e-300, s)
    return float(np.max(np.abs(a - b) / s))


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_zones,n_bins,n_lines", [(1, 300, 4000), (9, 7, 3000), (33, 65, 20000), (700, 20, 500),
                                                    (5, 2049, 8000)])
def test_opacity_shapes_match_oracle(sed_lib, precision, n_zones, n_bins, n_lines):
    w = workloads.type_ia(n_packets=10, n_zones=n_zones, n_lines=n_lines, n_bins=n_bins, bound_free=1,
                          n_levels_per_ion=7) if n_zones > 1 else _one_zone(n_bins, n_lines)
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    for e in (o, g):
        e.set_opacity(1.0)
    Oo, Og = o.opacity(), g.opacity()
    tol = 1e-12 if precision == abi.PREC_FP64 else 1e-5
    assert _maxrel(Og["n_elec"], Oo["n_elec"]) <= 1e-12
    for k in ("abs", "scat", "planck_mean", "rosseland_mean", "L_thermal"):
        assert _maxrel(Og[k], Oo[k]) <= tol, k
    assert np.max(np.abs(Og["emis_cdf"] - Oo["emis_cdf"])) <= tol  # CDF entries lie in [0, 1]
    o.close()
    g.close()


def _one_zone(n_bins, n_lines):
    w = workloads.type_ia(n_packets=10, n_zones=2, n_lines=n_lines, n_bins=n_bins, bound_free=1, n_levels_per_ion=7)
    z = w.zones
    for k in ("rho", "T", "X", "vol", "r_out", "v"):
        setattr(z, k, getattr(z, k)[1:])
    return w


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_levels", [100, 200, 250])
def test_long_level_lists_match_oracle(sed_lib, precision, n_levels):
    """Level lists around the shared-memory limit of the warp-per-zone LTE
    solve (3006, 6006 and 7506 levels): the last takes one thread per zone in
    both forms, the second in FP64."""
    w = workloads.type_ia(n_packets=10, n_zones=6, n_lines=500, n_bins=40, n_levels_per_ion=n_levels)
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    for e in (o, g):
        e.set_opacity(1.0)
    Oo, Og = o.opacity(), g.opacity()
    assert _maxrel(Og["n_elec"], Oo["n_elec"]) <= 1e-12
    for k in ("abs", "scat"):
        assert _maxrel(Og[k], Oo[k]) <= (1e-12 if precision == abi.PREC_FP64 else 1e-5), k
    o.close()
    g.close()


def test_fp64_lte_solve_is_the_same_in_both_forms(sed_lib, monkeypatch):
    """68 921 cells solved in one chunk (a thread per zone) and in small chunks
    (a warp per zone): the electron densities and tables are equal to the bit."""
    w = workloads.cart3d(n_packets=10, n_cells=41, n_lines=50, n_bins=4, n_levels_per_ion=5)
    out = []
    for scratch in (None, str(32 << 20)):
        if scratch:
            monkeypatch.setenv("SEDONA_GPU_OPACITY_SCRATCH_BYTES", scratch)
        g = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_FP64)
        g.set_opacity(1.0)
        out.append(g.opacity())
        g.close()
    for k in ("n_elec", "abs", "scat", "emis_cdf"):
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n_bins", [2, 33, 300, 1025])
def test_guide_tables_of_a_build_and_of_a_load_agree(sed_lib, precision, n_bins):
    """Packets on the tables of a build and on the same tables loaded back
    (whose guide tables the host forms by binary search) have the same
    histories to the bit."""
    n = 1500
    w = workloads.type_ia(n_packets=n, n_zones=20, n_lines=3000, n_bins=n_bins, seed=5)
    a = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    b = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
    a.set_opacity(1.0)
    t = a.opacity()
    b.load_opacity(t["abs"], t["scat"], t["emis_cdf"], t["eps_imc"])
    r = []
    for e in (a, b):
        e.record(True)
        e.transport(1.0)
        r.append(e.records(n))
        e.close()
    for k in ("fate", "ind", "draws", "state"):
        assert np.array_equal(r[0][k], r[1][k]), k
