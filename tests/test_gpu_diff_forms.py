"""Differentiable transport on FP32 tables against the oracle on the same
tables, around what its kernels choose by size: absorption depths on both sides
of the attenuation series' end, bands that do not divide the bins, one band per
bin, packets around the lanes of a warp, and replays repeated on one forward."""
import numpy as np
import pytest

from pubsed_b200 import abi, workloads
from pubsed_b200.adjoint import DiffEngine
import oracle_lib

pytestmark = pytest.mark.gpu


def _w(n, n_bins=90, epsilon=1e-3, **kw):
    return workloads.type_ia(n_packets=n, n_zones=14, n_lines=1500, n_bins=n_bins, spectrum_bins=24, epsilon=epsilon,
                             radiative_eq=0, seed=61, **kw)


@pytest.mark.parametrize("n,n_bins,n_bands,epsilon,scale", [(7, 90, 1, 1e-3, 1.0), (900, 90, 7, 1e-3, 1.0),
                                                           (900, 64, 64, 0.3, 1.0), (900, 90, 16, 0.05, 3.0),
                                                           (900, 90, 16, 0.05, 0.0)])
def test_forward_is_the_attenuated_path(sed_lib, n, n_bins, n_bands, epsilon, scale):
    """Scaling the absorption does not move a path, and every escaping energy is
    the unscaled one times exp(-(theta - 1) tau_a) of its path: three forwards
    at theta = 0, s and 2 s give log-energies on a line."""
    e = DiffEngine(_w(n, n_bins, epsilon), n_bands=n_bands, precision=abi.PREC_MIXED)
    e.tables()
    e.L.sed_record_packets(e.ctx, 1)
    st = []
    for th in (0.0, scale, 2 * scale):
        e.forward(np.full((e.nz, n_bands), th), step=2)
        st.append(_records(e, n))
    for r in st[1:]:
        for k in ("fate", "ind", "draws"):
            assert np.array_equal(r[k], st[0][k]), k
        assert np.array_equal(np.delete(r["state"], 7, axis=1), np.delete(st[0]["state"], 7, axis=1))
    l = [np.log(r["state"][:, 7]) for r in st]
    # two rounded attenuations per segment, at most 2^-52 each, over a few hundred segments, and the log's ulp
    assert np.all(np.abs((l[2] - l[1]) - (l[1] - l[0])) <= 1e-12 * (1 + np.abs(l[2]) + np.abs(l[0])))


@pytest.mark.parametrize("n,n_bands", [(7, 1), (900, 7), (3000, 90)])
def test_replay_matches_differences_and_repeats(sed_lib, n, n_bands):
    """The absorption gradient against the exact derivative of the exponential
    weights by central differences (paths fixed, so the only error is the
    difference's h^2), twice on the same forward."""
    e = DiffEngine(_w(n), n_bands=n_bands, precision=abi.PREC_MIXED)
    e.tables()
    g = np.linspace(0.5, 1.5, e.nspec)
    th = np.full((e.nz, n_bands), 0.9)
    e.forward(th, step=4)
    v = e.vjp(g)
    again = e.vjp(g)
    assert np.allclose(v, again, rtol=1e-12, atol=1e-12 * np.abs(v).max())
    d = np.linspace(-1.0, 1.0, th.size).reshape(th.shape)
    h = 1e-4
    f = [(g * e.forward(th + s * h * d, step=4)[0]).sum() for s in (1, -1)]
    fd = (f[0] - f[1]) / (2 * h)
    scale = np.abs(v * d).sum()
    assert abs(fd - (v * d).sum()) <= 1e-6 * scale
    e.close()


def _records(e, n):
    fate = np.zeros(n, np.int32); ind = np.zeros(n, np.int32); draws = np.zeros(n, np.int32)
    s = np.zeros(n * 9)
    rc = e.L.sed_get_packet_records(e.ctx, n, fate.ctypes.data_as(abi._ip), ind.ctypes.data_as(abi._ip),
                                    draws.ctypes.data_as(abi._ip), s.ctypes.data_as(abi._dp))
    assert rc == 0
    return {"fate": fate, "ind": ind, "draws": draws, "state": s.reshape(n, 9)}
