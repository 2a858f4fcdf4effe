"""The packet kernels' frequency-bin lookup on grids where its FP32 index
estimate is coarse: many bins over a narrow range, bins no float can tell
apart, linear grids far from zero, walls that do not follow min and del."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.grids import lin_grid, log_grid
import oracle_lib

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_lookup_gives_the_walls_bin(sed_lib, tmp_path):
    so = str(tmp_path / "bin_lookup.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "--fmad=false", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-o", so, os.path.join(HERE, "bin_lookup.cu")], check=True)
    f = C.CDLL(so).bin_lookup
    f.argtypes = [C.c_int, C.c_int, C.c_double, C.c_double, C.c_void_p, C.c_ulonglong, C.c_void_p]
    log = lambda ratio, n: log_grid(6e14, 6e14 * ratio, ratio ** (1.0 / n) - 1.0)
    grids = [log(100, 4096), log(1.02, 4096), log(1.01, 2000), log(1.005, 1000), log(1.0001, 300), log(1.5, 60000),
             log(1e6, 37), lin_grid(1e14, 1e16, 2.4e12), lin_grid(1e15, 1.001e15, 1e9), lin_grid(1e15, 1.0000001e15, 1e6),
             lin_grid(1e30, 1e40, 1.1e38)]
    bent = log(100, 500)
    bent.right = bent.right.copy()
    bent.right[:-1] *= 1 + 0.002 * np.sin(np.arange(bent.n - 1))
    for g in grids + [bent]:
        bad = np.zeros(1, np.uint64)
        r = np.ascontiguousarray(g.right)
        assert f(g.type, g.n, g.min, g.delta, r.ctypes.data, 1 << 24, bad.ctypes.data) == 0
        assert bad[0] == 0, (g.type, g.n, g.min, g.delta, bad[0])


def test_packets_on_a_narrow_grid_match_oracle(sed_lib):
    """FP64 packets through line opacity in 4096 bins over 2 % in frequency have
    the oracle's histories to the bit."""
    n = 250
    w = workloads.type_ia(n_packets=n, n_zones=12, n_lines=400_000, n_bins=256, spectrum_bins=16, seed=3)
    lo, hi = 6e14, 6.12e14
    w.params["transport_nu_grid"] = [lo, hi, workloads.log_delta_for_bins(lo, hi, 4096), 1]
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(sed_lib, "sed_", w)
    o.set_opacity(1.0)
    t = o.opacity()
    assert np.unique(t["abs"].reshape(12, -1)[6]).size > 1000
    r = []
    for e in (o, g):
        e.load_opacity(t["abs"], t["scat"], t["emis_cdf"], t["eps_imc"])
        e.record(True)
        e.transport(1.0)
        r.append(e.records(n))
        e.close()
    for k in ("fate", "ind", "draws"):
        assert np.array_equal(r[0][k], r[1][k]), k
    oracle_lib.check_states(r[1]["state"], r[0]["state"])
