"""gz_density_sums_noalloc where its runs, tiles and hit lists have their edges: set sizes around a run of 32
particles, a block's tile and the limit; targets whose kernels reach far more particles than their neighbours'
(the cross-lane evaluation), coincident particles, kernels across the periodic faces, and positions and kernels
that no FP32 screen may reject. Against gz_density_sums, which takes the same terms in another order."""
import ctypes as C

import numpy as np
import pytest

from gizmo_b200 import abi, ics
from gizmo_b200.hydro import HydroPass

pytestmark = pytest.mark.gpu


def _noalloc(wl):
    import torch

    dev = torch.device("cuda", 0)
    d = {k: torch.as_tensor(np.ascontiguousarray(getattr(wl, k)), device=dev) for k in ("pos", "vel", "mass", "h")}
    acc = torch.full((wl.n, 14), float("nan"), dtype=torch.float64, device=dev)
    pv = torch.full((wl.n, 3), float("nan"), dtype=torch.float64, device=dev)
    s = torch.cuda.current_stream(dev)
    rc = abi.load_library().gz_density_sums_noalloc(
        C.byref(wl.params), wl.n, *(d[k].data_ptr() for k in ("pos", "vel", "mass", "h")), acc.data_ptr(), pv.data_ptr(),
        C.c_void_p(s.cuda_stream))
    assert rc == abi.OK
    s.synchronize()
    return acc.cpu().numpy(), pv.cpu().numpy()


def _subset(n, seed=4):
    wl = ics.plummer_mix(41, seed=seed, n_spheres=12)
    for k in ("pos", "vel", "mass", "u", "dt", "h", "cond"):
        setattr(wl, k, np.ascontiguousarray(getattr(wl, k)[:n]))
    wl.h = wl.h * (68921 / n) ** (1 / 3)  # the same neighbour count in the thinned set
    wl.h = np.minimum(wl.h, 0.2)
    return wl


def _check(wl):
    with HydroPass(wl.params) as hp:
        hp.upload_workload(wl)
        want, want_pv = hp.density_sums()
    acc, pv = _noalloc(wl)
    # Two orders of a sum of N terms differ by at most 2 N 2^-53 sum|term|: 1e-12 of that scale covers N = 4500.
    # sum|term| from the sums of positive terms: a0 = sum W holds the target's own W(0) = 8 / (pi h^3) (Wendland
    # C2: 3.3 / h^3), and |dW| h, |u dW| h are below that each, so 100 a0 / h bounds theirs for N up to 100 (and
    # a0 grows with N beyond).
    h, a0, v = wl.h, want[:, 0], 2 * np.abs(wl.vel).max()
    scale = [a0, want[:, 1], 100 * a0 / h, 100 * v * a0 / h] + [h * h * a0] * 6 + [h * a0] * 3
    for c, sc in enumerate(scale):
        assert (np.abs(acc[:, c] - want[:, c]) <= 1e-12 * sc).all(), (c, np.max(np.abs(acc[:, c] - want[:, c]) / sc))
    assert (acc[:, 13] == 0).all()
    assert (np.abs(pv - want_pv) <= 1e-12 * v * want[:, 1:2]).all()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 4097, 20001, 65536])
def test_sizes(n):
    _check(_subset(n))


@pytest.mark.parametrize("field", ["lone", "all", "coincident"])
def test_uneven_and_long_kernels(field):
    wl = _subset(3000)
    if field == "lone":  # one target in a hundred reaches hundreds of particles, the rest a few
        wl.h[::100] = 0.25
    elif field == "all":  # every pair of the set
        wl = _subset(500)
        wl.h[:] = 0.4999
    else:
        wl.pos[1000:1040] = wl.pos[1000]
        wl.pos[:3] = [[0.0, 0.5, 0.5], [1.0 - 2.0 ** -53, 0.5, 0.5], [1e-9, 0.5, 0.5]]
    _check(wl)


def test_a_nan_position_reaches_every_sum():
    """A pair with a NaN separation is not outside any kernel (r2 >= h2 is false), so it enters every target's sums."""
    wl = _subset(1000)
    wl.pos[500, 1] = np.nan
    acc, _ = _noalloc(wl)
    assert np.isnan(acc[:, 0]).all()


@pytest.mark.parametrize("shift", [-200, -70, 70, 200])
def test_the_unit_of_length_does_not_matter(shift):
    """Lengths scaled by a power of two scale every sum by one: no rounding differs, so neither does any decision of
    the screen. (At 2^-70 the squares of FP32 separations would be denormal, at 2^70 infinite.)"""
    import copy

    want = _subset(3000)
    wl = copy.deepcopy(want)
    f = 2.0 ** shift
    wl.pos, wl.h, wl.params.box_size = wl.pos * f, wl.h * f, want.params.box_size * f
    a, apv = _noalloc(want)
    b, bpv = _noalloc(wl)
    # W, m W ~ 1 / h^3; 3 W / h + u dW/du and dW/dr dx dv / r ~ 1 / h^4; x x W ~ 1 / h; x W ~ 1 / h^2
    for c, power in enumerate([3, 3, 4, 4] + [1] * 6 + [2] * 3):
        assert np.array_equal(b[:, c] * f ** power, a[:, c]), c
    assert np.array_equal(bpv * f ** 3, apv)
