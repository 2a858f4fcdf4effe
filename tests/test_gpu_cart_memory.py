"""A 3D mixed step takes per-packet emission slots only where they leave room:
with little memory free it emits in the packet kernel, and the packets are the
same."""
import numpy as np
import pytest

from pubsed_b200 import abi
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


def test_little_memory_leaves_the_slots_out(sed_lib):
    import torch

    n, slots = 4_000_000, 4_000_000 * 76
    w = grey_box(n, shape=(6, 5, 4), seed=9, radiative_eq=0)
    w.params["opacity_grey_opacity"] = 1e-3  # thin: the step is short
    e = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    e.set_opacity(1.0)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - 2 * slots + (64 << 20), dtype=torch.uint8, device="cuda")
    try:
        before = torch.cuda.mem_get_info()[0]
        assert slots < before < 2 * slots
        a = e.transport(1.0)
        assert torch.cuda.mem_get_info()[0] > before - slots // 2
        few = e.spectrum()
    finally:
        del filler
        torch.cuda.empty_cache()
    e.check(sed_lib.sed_set_rng_step(e.ctx, 0), "set_rng_step")
    b = e.transport(1.0)
    assert torch.cuda.mem_get_info()[0] < free - slots // 2  # the slots are there
    much = e.spectrum()
    for k in ("n_escaped", "n_absorbed", "n_segments", "n_scatters"):
        assert a[k] == b[k], k
    assert np.array_equal(few[1], much[1])
    assert np.allclose(few[0], much[0], rtol=1e-11, atol=0)
    e.close()
