"""The packed bins of the 1D mixed kernel are taken only where they leave room:
a context that fits without them is made without them, and its packets are the
same."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib

pytestmark = pytest.mark.gpu


def test_a_context_that_fits_without_them_is_made(sed_lib):
    import torch

    n, zones, bins = 3000, 2000, 4096
    packed = 16 * zones * bins
    w = workloads.lightbulb_grey(n_packets=n, n_zones=zones, n_bins=bins, radiative_eq=1, seed=5)
    w.params["spectrum_nu_grid"] = [1e14, 1e16, workloads.log_delta_for_bins(1e14, 1e16, 32), 1]

    def run(e):
        e.set_opacity(1.0)
        e.record(True)
        e.transport(1.0)
        return e.records(n)

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    def context():
        return oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)

    first = context()  # the kernels are loaded
    a = run(first)
    first.close()
    before = free()
    e = context()
    need = before - free()
    e.close()
    assert need > 2 * packed
    filler = torch.empty(free() - (need - packed) - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        e = context()
        b = run(e)
    finally:
        del filler
        torch.cuda.empty_cache()
    for k in ("fate", "ind", "draws", "state"):
        assert np.array_equal(a[k], b[k]), k
    e.close()
