"""Symmetric rows of an active list, taken in one walk (rows in slots, then copied to their places; rows longer than
their slots filled by a walk of their own), against the oracle's exact search: lists that take the walk's two modes,
their shortest lengths, and slots too short for every row, for some and for none."""
import numpy as np
import pytest

from gizmo_b200 import ics
from gizmo_b200.hydro import HydroPass
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1.0, 2.5, 16.0])
@pytest.mark.parametrize("k", [1, 2, 33, 1500, 12000])
def test_rows_of_active_lists(k, slots):
    wl = ics.plummer_mix(24, seed=4, n_spheres=10)
    rng = np.random.default_rng(k)
    act = np.sort(rng.choice(wl.n, size=k, replace=False)).astype(np.int32)
    with HydroPass(wl.params) as hp:
        hp.set_tuning(96, slots)
        hp.upload_workload(wl)
        hp.full_pass()
        full = hp.download(["h", "grad_rho", "grad_v"])
        hp.hydro_gradient_calc(act)
        rows = hp.status()["pairs_symmetric"]
        sub = hp.download(["h", "grad_rho", "grad_v"])
    st = O.new_state(wl.n, wl.inputs())
    st["h"][:] = full["h"]
    off, _ = O.neighbors(wl.params, st, 1)
    assert rows == int((off[act + 1] - off[act]).sum())
    # the same neighbours in another number of lanes: summation order only (as the parity tests bound it)
    for f in ("grad_rho", "grad_v"):
        a, b = sub[f][act], full[f][act]
        assert (np.linalg.norm(a - b, axis=1) <= 1e-10 * np.maximum(np.linalg.norm(b, axis=1), 1e-6 * np.abs(full[f]).max())).all()
