"""The FP64 packet kernel of homologous grids: its branch-free divisions and
roots against CUDA's, and packets against the oracle over the forms the kernel
takes (grids, bins, switches, packet counts around the lanes of a warp)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_ieee_sequences_equal_cudas(sed_lib, tmp_path):
    so = str(tmp_path / "fp64_ops.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "fp64_ops.cu")], check=True)
    f = C.CDLL(so).fp64_ops
    f.argtypes = [C.c_void_p, C.c_ulonglong, C.c_int, C.c_int, C.c_double]
    for lo, hi, t in ((-1, 1, 864000.0), (-60, 90, 1.728e6), (-300, 300, 3.1e7), (0, 52, 1.0000000000000002)):
        bad = np.zeros(7, np.uint64)
        assert f(bad.ctypes.data, 1 << 26, lo, hi, t) == 0
        assert not bad.any(), (lo, hi, t, bad)


def _bulb(n, n_bins=60, radiative_eq=1, n_zones=11, **params):
    w = workloads.lightbulb_grey(n_packets=n, n_zones=n_zones, n_bins=n_bins, radiative_eq=radiative_eq, seed=13)
    w.params.update(params)
    return w


def _check(w, n):
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(oracle_lib_sed(), "sed_", w)
    for e in (o, g):
        e.set_opacity(1.0)
        e.record(True)
    so, sg = o.transport(1.0), g.transport(1.0)
    ro, rg = o.records(n), g.records(n)
    for k in ("fate", "ind", "draws"):
        assert np.array_equal(ro[k], rg[k]), k
    oracle_lib.check_states(rg["state"], ro["state"])
    for k in ("n_escaped", "n_absorbed", "n_stopped", "n_segments", "n_scatters"):
        assert so[k] == sg[k], k
    fo, co = o.spectrum()
    fg, cg = g.spectrum()
    assert np.array_equal(co, cg)
    To, Tg = o.tallies(), g.tallies()
    for k in ("J_nu", "e_abs"):
        oracle_lib.zone_tally_close(Tg[k], To[k])
    o.close()
    g.close()


def oracle_lib_sed():
    from pubsed_b200 import _lib
    return _lib.lib()


CORE = 0.3 * 1e9 * 864000.0
FORMS = {
    "few": dict(n=3), "a warp and one": dict(n=33), "two bins": dict(n=400, n_bins=2), "one zone": dict(n=500, n_zones=1),
    "no equilibrium": dict(n=800, radiative_eq=0), "absorbing core": dict(n=800, core_radius=CORE),
    "reflecting core": dict(n=300, core_radius=CORE, transport_boundary_in_reflect=1),
    "reflecting edge": dict(n=200, radiative_eq=0, transport_boundary_out_reflect=1),
    "no scattering": dict(n=500, opacity_no_scattering=1), "no J": dict(n=500, transport_store_Jnu=0),
    "linear bins": dict(n=400, transport_nu_grid=[1e14, 1e16, 2e13], spectrum_nu_grid=[1e14, 1e16, 2e13]),
    "one frequency": dict(n=400, core_photon_frequency=7e14),
}


@pytest.mark.parametrize("form", sorted(FORMS))
def test_sphere_forms_match_oracle(sed_lib, form):
    k = dict(FORMS[form])
    n = k.pop("n")
    _check(_bulb(n, **k), n)


@pytest.mark.parametrize("n,radiative_eq", [(1, 1), (700, 0), (2500, 1)])
def test_cartesian_forms_match_oracle(sed_lib, n, radiative_eq):
    _check(grey_box(n, shape=(3, 1, 6), seed=5, radiative_eq=radiative_eq), n)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
def test_packet_counts_share_histories(sed_lib, precision):
    """Runs of 5, 2500 (one packet per warp, then two) and 80 000 packets (all
    lanes) give the packets they share the same histories to the bit (all of
    the state but the packet's energy, which is the luminosity over n)."""
    out = []
    for n in (5, 2500, 80_000):
        w = workloads.type_ia(n_packets=n, n_zones=20, n_lines=2000, n_bins=200, spectrum_bins=16, seed=3)
        g = oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)
        g.set_opacity(1.0)
        g.record(True)
        g.transport(1.0)
        r = g.records(n)
        r["state"] = np.delete(r["state"], 7, axis=1)
        out.append(r)
        g.close()
    for a, m in ((out[0], 5), (out[1], 2500)):
        for k in ("fate", "ind", "draws", "state"):
            assert np.array_equal(a[k][:m], out[2][k][:m]), k
            assert np.array_equal(out[0][k], out[1][k][:5]), k
