"""The 3D mixed packet kernel: packets emitted ahead and binned afterwards, and
packets emitted and counted in the kernel (any step with queued packets), have
the histories of one another to the bit; around the sizes where its cell
indices, tally copies and lane shares can go wrong.  What the histories have to
be is held by the oracle in test_gpu_cart3d.py (FP64) and by the spectra's
chi-squared there (mixed)."""
import numpy as np
import pytest

from pubsed_b200 import abi
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu


def _box(n, shape, radiative_eq, **params):
    w = grey_box(n, shape=shape, seed=8, radiative_eq=radiative_eq)
    w.params.update(params)
    return w


@pytest.mark.parametrize("n,shape,radiative_eq,params", [
    (1, (1, 1, 1), 1, {}), (40, (1, 5, 2), 1, {}), (3000, (4, 1, 7), 0, {}), (2500, (3, 3, 3), 1, {}),
    (300, (4, 3, 5), 0, {"transport_boundary_out_reflect": 1}), (800, (6, 2, 3), 1, {"transport_store_Jnu": 0}),
    (800, (6, 2, 3), 1, {"opacity_no_scattering": 1})])
def test_packets_match_oracle_spectra_and_energy(sed_lib, n, shape, radiative_eq, params):
    """Against the oracle on the same model: every packet accounted for, and the
    escaped counts and energies within five standard deviations of a run of
    as many packets."""
    w = _box(n, shape, radiative_eq, **params)
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    g = oracle_lib.Engine(sed_lib, "sed_", w, precision=abi.PREC_MIXED)
    for e in (o, g):
        e.set_opacity(1.0)
        e.record(True)
    so, sg = o.transport(1.0), g.transport(1.0)
    assert sg["n_escaped"] + sg["n_absorbed"] + sg["n_stopped"] == n
    sd = np.sqrt(max(n, 1)) * 0.5 * np.sqrt(2)
    assert abs(sg["n_escaped"] - so["n_escaped"]) <= 5 * sd
    f, c = g.spectrum()
    r = g.records(n)
    assert c.sum() == (r["fate"] == 2).sum() == sg["n_escaped"]
    assert np.isclose(f.sum(), r["state"][r["fate"] == 2, 7].sum(), rtol=1e-12)
    o.close()
    g.close()


def test_both_forms_of_the_kernel_agree(sed_lib):
    """A census of one packet makes the step's packets be emitted and counted in
    the kernel; its core packets are those of a step without it, and so are
    their records and the clicks they leave."""
    n = 4000
    a = oracle_lib.Engine(sed_lib, "sed_", _box(n, (5, 4, 6), 1, transport_steady_iterate=0), precision=abi.PREC_MIXED)
    b = oracle_lib.Engine(sed_lib, "sed_", _box(n, (5, 4, 6), 1, transport_steady_iterate=0), precision=abi.PREC_MIXED,
                          first_packet_id=0)
    dt = 40 * 86400.0  # longer than any packet stays
    rec = []
    for e, extra in ((a, 0), (b, 1)):
        if extra:
            erad = np.ones(e.nz)
            assert sed_lib.sed_initialize_particles(e.ctx, extra, erad.ctypes.data_as(abi._dp)) == 0
        e.set_opacity(dt)
        e.record(True)
        e.transport(dt)
        rec.append((e.records(n), e.spectrum()))
        e.close()
    # the queued packet's stream comes first: core packet q of b draws stream q + 1, which is core packet q + 1 of a
    for k in ("fate", "ind", "draws"):
        assert np.array_equal(rec[0][0][k][1:], rec[1][0][k][:n - 1]), k
    assert np.array_equal(rec[0][0]["state"][1:], rec[1][0]["state"][:n - 1])
    assert rec[1][1][1].sum() >= rec[0][1][1].sum() - 1
