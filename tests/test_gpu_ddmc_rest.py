"""Discrete diffusion on a static sphere, on one whose outer zones move, and
with a hollow centre: zones at rest skip the transforms, and every zone's
leakage factors come from the step's table, against the oracle's packets."""
import numpy as np
import pytest

from pubsed_b200 import workloads
import oracle_lib

pytestmark = pytest.mark.gpu


def _steps(eng, w, n, dt, steps):
    eng.initialize_particles(n, workloads.initial_e_rad(w.zones))
    out = []
    for _ in range(steps):
        eng.set_opacity(dt)
        eng.record(True)
        st = eng.transport(dt)
        out.append({"stats": st, "records": eng.records(st["n_packets"]), "census": eng.census(),
                    "tallies": eng.tallies(), "spectrum": eng.spectrum()})
    return out


@pytest.mark.parametrize("v_outer,r_min,n_zones,tau", [
    (0.0, 0.0, 200, 0.1), (0.0, 5.25, 40, 0.6), (2e8, 0.0, 40, 0.1), (2e8, 0.0, 40, 0.6)])
def test_static_and_moving_zones(sed_lib, v_outer, r_min, n_zones, tau):
    def model():
        w = workloads.diffusing_pulse(n_initialize=4000, seed=31)
        r = r_min + 0.5 * (1 + np.arange(n_zones))
        z = w.zones
        z.r_min, z.r_out, z.rho = r_min, r, 1.0 + 0.5 * np.sin(np.arange(n_zones))
        z.T = np.where(np.arange(n_zones) < 10, 1e4, 0.0)
        z.X = np.ones((n_zones, 1))
        z.vol = workloads.shell_volumes(r_min, r)
        z.v = np.where(np.arange(n_zones) < n_zones // 2, 0.0, v_outer * r / r[-1])
        w.params["transport_ddmc_tau_threshold"] = tau
        return w
    runs = []
    for lib, prefix in ((sed_lib, "sed_"), (oracle_lib.oracle_lib(), "oracle_")):
        w = model()
        e = oracle_lib.Engine(lib, prefix, w)
        runs.append(_steps(e, w, 4000, 2e-10, 3))
        e.close()
    oracle_lib.compare_td(*runs)
