"""The LTE solve on either side of the lines between its forms (a warp or a
thread per zone), with short level lists: against the oracle, and in FP64 the
two forms against each other to the bit."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib

pytestmark = pytest.mark.gpu


def _model(cells, atoms, levels):
    """A clumped 3D model of the first `atoms` elements."""
    w = workloads.cart3d(n_packets=10, n_cells=cells, n_lines=60, n_bins=4, n_levels_per_ion=levels)
    z = w.zones
    X = z.X[:, :atoms] + 1e-3
    z.X = np.ascontiguousarray(X / X.sum(1, keepdims=True))
    z.elem_Z, z.elem_A = z.elem_Z[:atoms], z.elem_A[:atoms]
    w.atoms.atoms = w.atoms.atoms[:atoms]
    return w


# 148 SMs: lines at 18 944 zones, at 64 levels with FP32 tables and at 210 zones per level in FP64
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("cells,atoms,levels", [(26, 1, 2), (27, 1, 2), (27, 1, 12), (27, 1, 14), (27, 2, 10), (32, 6, 5)])
def test_electron_densities_match_oracle(sed_lib, precision, cells, atoms, levels):
    w = _model(cells, atoms, levels)
    ne = []
    for lib, prefix, p in ((oracle_lib.oracle_lib(), "oracle_", abi.PREC_FP64), (sed_lib, "sed_", precision)):
        e = oracle_lib.Engine(lib, prefix, w, precision=p)
        e.set_opacity(1.0)
        ne.append(e.opacity()["n_elec"])
        e.close()
    assert np.all(ne[0] > 0)
    assert np.max(np.abs(ne[1] - ne[0]) / ne[0]) <= 1e-12


def test_forms_agree_to_the_bit(sed_lib, monkeypatch):
    """FP64, 19 683 zones: a thread each in one chunk, a warp each in small ones."""
    w = _model(27, 2, 5)
    out = []
    for scratch in (None, str(8 << 20)):
        if scratch:
            monkeypatch.setenv("SEDONA_GPU_OPACITY_SCRATCH_BYTES", scratch)
        g = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_FP64)
        g.set_opacity(1.0)
        out.append(g.opacity())
        g.close()
    for k in ("n_elec", "abs", "scat", "emis_cdf"):
        assert np.array_equal(out[0][k], out[1][k]), k
