"""The emissivity CDF of the blocked scan (FP32 tables, and FP64 grids of many
zones): like the sequential sum it stands for, a row never falls and ends at 1,
also where most bins emit next to nothing."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("cells,n_bins", [(41, 33), (41, 300), (20, 2048)])
def test_rows_never_fall(sed_lib, precision, cells, n_bins):
    w = workloads.cart3d(n_packets=10, n_cells=cells, n_lines=2000, n_bins=n_bins, n_levels_per_ion=5)
    e = Engine(w, precision=precision)
    e.set_opacity(1.0)
    cdf = e.opacity()["emis_cdf"].reshape(cells ** 3, n_bins)
    e.close()
    assert np.all(cdf >= 0)
    assert np.count_nonzero(np.diff(cdf, axis=1) < 0) == 0
    assert np.all(cdf[:, -1] == 1.0)
