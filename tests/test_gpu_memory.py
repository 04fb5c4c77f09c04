"""Device memory near its limit. The tests fill the GPU with a torch allocation, so that a context finds only as much
free memory as they leave; every failure is an answer of cudaMalloc on the host."""
import contextlib

import numpy as np
import pytest

from gizmo_b200 import abi, ics
from gizmo_b200.hydro import GizmoHydroError, HydroPass

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _only_free(nbytes):
    """All of the device's memory but nbytes, and 12 MB at most beyond, taken while the context is open. (The caching
    allocator takes exact multiples of 2 MB from the device for what is larger than 10 MB, 20 MB for what is smaller.)"""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    while (excess := torch.cuda.mem_get_info()[0] - nbytes) >= 12 * MB:
        held.append(torch.empty(min(excess, 1 << 36) // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _uniform(n, seed=1):
    rng = np.random.default_rng(seed)
    one = np.ones(n)
    return dict(pos=rng.random((n, 3)), vel=np.zeros((n, 3)), mass=one / n, u=one, dt=one * 2.0 ** -8,
                h=one * (32 / (4.19 * n)) ** (1 / 3))


def test_a_failed_allocation_reports_cudas_own_words_and_can_be_repeated():
    wl = ics.sedov(12)
    big = _uniform(2_000_000)
    with HydroPass(wl.params) as hp:
        hp.upload_workload(wl)
        hp.full_pass()
        want = hp.download()
        with _only_free(100 * MB):
            with pytest.raises(GizmoHydroError, match="cudaMalloc of [0-9]+ bytes: out of memory"):
                hp.upload(**big)
        # the set is lost with its buffers: what needs one is refused, and a download has nothing to bring
        for call in (hp.density, hp.hydro_gradient_calc, hp.hydro_force, lambda: hp.neighbors(0)):
            with pytest.raises(GizmoHydroError) as e:
                call()
            assert e.value.code == abi.ERR_ORDER
        hp.upload_workload(wl)
        hp.full_pass()
        got = hp.download()
        for k in want:
            assert np.array_equal(got[k], want[k]), k


def _crept(precision, n=600_000):
    """A context whose pair buffers have grown by a little and hold room to grow further, with its last results."""
    p = ics.sedov(4, precision=precision).params
    hp = HydroPass(p)
    hp.upload(**_uniform(n))
    hp.full_pass()
    p.des_num_ngb = 33.0
    hp.set_params(p)
    hp.restage()
    hp.full_pass()
    return hp, hp.status()


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_room_to_grow_is_given_back_before_an_allocation_fails(precision):
    n = 600_000
    flux = {abi.PRECISION_FP64: 64, abi.PRECISION_MIXED: 32}[precision]
    names = ["h", "rho", "accel", "dudt"]
    hp, _ = _crept(precision, n)
    with hp:
        want = hp.download(names)
    hp, st = _crept(precision, n)  # (a download takes staging: this one has made none)
    with hp:
        sized = hp.status()["device_bytes"]
        room = flux * st["pairs_symmetric"] // 4  # what the fluxes hold beyond their entries, at least
        assert room > 16 * 8 * n
        # free: too little for a download's staging (16 doubles a particle)
        with _only_free(40 * MB):
            got = hp.download()
            assert hp.status()["device_bytes"] < sized
            for k in names:
                assert np.array_equal(got[k], want[k]), k
            # and the pass itself still runs, in buffers of the exact sizes
            hp.restage()
            hp.full_pass()
            got = hp.download(names)
            for k in names:
                assert np.array_equal(got[k], want[k]), k


def test_rows_left_to_the_force_pass_survive_a_lack_of_memory():
    """Gradients, then a download that has to find its staging in the rows' spare room, then the force on those rows."""
    hp, _ = _crept(abi.PRECISION_FP64)
    with hp:
        want = hp.download()
    hp, _ = _crept(abi.PRECISION_FP64)
    with hp:
        hp.restage()
        hp.density()
        hp.hydro_gradient_calc()
        with _only_free(40 * MB):
            hp.download(["rho"])
            hp.hydro_force()
            got = hp.download(["accel", "dudt", "vsig"])
        for k in got:
            assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("graph", [False, True])
def test_fp64_force_without_room_for_the_fluxes(graph):
    """Each row then evaluates its pairs in place: the same terms in another order."""
    n = 300_000
    p = ics.sedov(4).params
    with HydroPass(p) as hp:
        hp.upload(**_uniform(n))
        hp.full_pass()
        want = hp.download()
        hp.download()
    with HydroPass(p) as hp:
        hp.upload(**_uniform(n))
        hp.density()
        hp.hydro_gradient_calc()
        hp.download()  # (its staging is held from here on)
        with _only_free(300 * MB):  # the fluxes take 64 bytes an entry, about 800 MB
            if graph:
                hp.hydro_pass(graph=True, restage=True)
                assert hp.graph_stats()["replays"] == 0
            else:
                hp.hydro_force()
            got = hp.download()
    for k in ("h", "rho", "grad_rho"):
        assert np.array_equal(got[k], want[k]), k
    for k in ("accel", "dudt", "vsig"):
        scale = np.abs(want[k]).max()
        assert np.abs(got[k] - want[k]).max() <= 1e-12 * scale, k


def test_mixed_force_with_room_for_the_fluxes_only():
    """The queue of the deferred pairs then has room for a few of them, and the rows are scanned for the others."""
    n = 600_000
    q = _uniform(n)
    q["vel"] = np.random.default_rng(2).standard_normal((n, 3)) * 2.0
    p = ics.sedov(4, precision=abi.PRECISION_MIXED).params
    got, names = {}, ["accel", "dudt", "vsig"]
    for where in ("roomy", "tight"):
        with HydroPass(p) as hp:
            hp.upload(**q)
            hp.density()
            hp.hydro_gradient_calc()
            hp.download(["h"])  # (its staging is held from here on)
            pairs = hp.status()["pairs_symmetric"]
            # fluxes 32 bytes an entry, the refine queue 32 for one in 8, the deferred pairs' queue 32 for one in 32;
            # the rows' scratch, 4 an entry, is given back for them
            with _only_free((32 + 4 - 4) * pairs + 6 * MB) if where == "tight" else contextlib.nullcontext():
                assert pairs > 16 * MB
                hp.hydro_force()
                deferred, room = hp.force_deferred()
                got[where] = hp.download(names)
            assert deferred > 1024 and (room == 1024) == (where == "tight"), (where, deferred, room)
    for k in names:
        assert np.array_equal(got["tight"][k], got["roomy"][k]), k


def test_a_set_that_creeps_up_is_not_allocated_anew_each_time():
    """Far from the device's limit; near it the buffers keep to their exact sizes."""
    p = ics.sedov(4).params
    n = 300_000
    a = _uniform(n + 40)
    part = lambda k: {f: v[:k] for f, v in a.items()}  # noqa: E731
    sizes = {}
    for where in ("roomy", "tight"):
        with HydroPass(p) as hp, _only_free(2000 * MB) if where == "tight" else contextlib.nullcontext():
            sizes[where] = []
            for k in (n, n + 10, n + 20, n + 30, n + 40):
                hp.upload(**part(k))
                hp.density()
                sizes[where].append(hp.status()["device_bytes"])
    assert sizes["roomy"][1] > 1.1 * sizes["roomy"][0]
    assert len(set(sizes["roomy"][1:])) == 1, sizes
    assert sizes["tight"][4] < 1.05 * sizes["tight"][0], sizes
