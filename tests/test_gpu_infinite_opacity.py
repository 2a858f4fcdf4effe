"""Opacities that are infinite: a black wall (absorption) ends a packet at its
first step into the zone, a white one (scattering) holds it there."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib
from test_gpu_cart3d import grey_box

pytestmark = pytest.mark.gpu
ABSORBED = 3  # sed_get_packet_records


def _model(kind, n):
    if kind == "box":
        return grey_box(n, shape=(5, 6, 4), seed=3, radiative_eq=0)
    w = workloads.lightbulb_grey(n_packets=n, n_zones=9, n_bins=50, radiative_eq=0, seed=3)
    if kind == "static sphere":
        w.zones.homologous = 0
        w.zones.v = np.zeros(9)
    return w


def _run(sed_lib, w, precision, n, key, limit=0):
    """Oracle's and library's records with the opacity `key` infinite in every
    third zone, and whether the run ended at the segment limit."""
    w.params["gpu_max_segments"] = limit
    o = oracle_lib.Engine(oracle_lib.oracle_lib(), "oracle_", w)
    o.set_opacity(1.0)
    t = o.opacity()
    nz, nn = o.nz, o.nn
    wall = np.arange(nz) % 3 == 2
    for k in ("abs", "scat"):
        a = t[k].reshape(nz, nn)
        a[wall] = np.inf if k == key else 0.0
    out = []
    for e in (o, oracle_lib.Engine(sed_lib, "sed_", w, precision=precision)):
        e.load_opacity(t["abs"], t["scat"], t["emis_cdf"], np.ones(nz))
        e.record(True)
        hit = False
        try:
            e.transport(1.0)
        except RuntimeError as err:
            hit = "segment limit" in str(err)
            assert hit
        out.append((e.records(n), hit))
        e.close()
    return wall, out


@pytest.mark.parametrize("kind", ["sphere", "static sphere", "box"])
def test_fp64_packets_end_at_a_black_wall(sed_lib, kind):
    n = 400
    wall, ((ro, _), (rg, _)) = _run(sed_lib, _model(kind, n), abi.PREC_FP64, n, "abs")
    assert np.count_nonzero((ro["fate"] == ABSORBED) & wall[np.clip(ro["ind"], 0, None)]) > n // 4
    for k in ("fate", "ind", "draws"):
        assert np.array_equal(ro[k], rg[k]), k
    oracle_lib.check_states(rg["state"], ro["state"])


@pytest.mark.parametrize("kind,precision", [("sphere", abi.PREC_FP64), ("static sphere", abi.PREC_FP64),
                                            ("box", abi.PREC_FP64), ("box", abi.PREC_MIXED)])
def test_packets_are_held_by_a_white_wall(sed_lib, kind, precision):
    n = 200
    wall, ((ro, ho), (rg, hg)) = _run(sed_lib, _model(kind, n), precision, n, "scat", limit=300)
    assert ho and hg
    for r in (ro, rg):
        inside = wall[np.clip(r["ind"], 0, None)] & (r["ind"] >= 0)
        assert np.count_nonzero(inside) > n // 10
        assert not np.any(r["fate"][inside] == ABSORBED)  # nothing absorbs there
    if precision == abi.PREC_FP64:
        for k in ("fate", "ind", "draws"):
            assert np.array_equal(ro[k], rg[k]), k
