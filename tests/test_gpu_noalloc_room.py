"""sed_lte_electron_density_noalloc with room for more stages and levels than
the lists hold: the lists decide, the counts only size the working set."""
import ctypes as C

import numpy as np
import pytest

from pubsed_b200 import abi, workloads
import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1, 40])
def test_room_beyond_the_lists_changes_nothing(sed_lib, more):
    import torch

    w = workloads.type_ia(n_packets=10, n_zones=30, n_lines=300, n_bins=16, n_levels_per_ion=5, seed=21)
    g = oracle_lib.Engine(sed_lib, "sed_", w)
    g.set_opacity(1.0)
    ref = g.opacity()["n_elec"]
    g.close()
    keep = abi.Keep()
    a = w.atomic_struct(keep)
    na = a.n_atoms
    host = lambda p, n: np.ctypeslib.as_array(p, shape=(n,)).copy()
    n_ions, n_levs = int(host(a.ion_off, na + 1)[na]), int(host(a.lev_off, na + 1)[na])
    z = w.zones
    t = [torch.from_numpy(x).cuda() for x in (
        host(a.ion_off, na + 1), host(a.ion_chi, n_ions), host(a.lev_off, na + 1), host(a.lev_ion, n_levs),
        host(a.lev_g, n_levs), host(a.lev_E, n_levs), z.rho.copy(), z.T.copy(), np.ascontiguousarray(z.X.reshape(-1)),
        z.elem_A.astype(np.int32))]
    ne = torch.zeros(z.n_zones, dtype=torch.float64, device="cuda")
    err = torch.full((z.n_zones,), -1, dtype=torch.int32, device="cuda")
    ad = abi.AtomicData()
    ad.n_atoms = na
    for k, x in zip(("ion_off", "ion_chi", "lev_off", "lev_ion", "lev_g", "lev_E"), t):
        setattr(ad, k, C.cast(x.data_ptr(), abi._dp if x.dtype == torch.float64 else abi._ip))
    f = sed_lib.sed_lte_electron_density_noalloc
    f.argtypes = [C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.POINTER(abi.AtomicData),
                  C.c_int32, C.c_int32, C.c_double, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    rho, T, X, A = (x.data_ptr() for x in t[6:])
    rc = f(z.n_zones, rho, T, X, z.n_elems, A, C.byref(ad), n_ions + more, n_levs + 2 * more,
           w.P.scalar("limits_temp_min"), w.P.scalar("limits_temp_max"), ne.data_ptr(), err.data_ptr(),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0 and np.all(err.cpu().numpy() == 0)
    assert np.array_equal(ne.cpu().numpy(), ref)
