"""Device memory near its limit. The tests fill the GPU with a torch allocation, so that a context finds only as much
free memory as they leave; every failure is an answer of cudaMalloc on the host."""
import contextlib

import numpy as np
import pytest

from gizmo_b200 import ics
from gizmo_b200.hydro import GizmoHydroError, HydroPass

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _only_free(nbytes):
    """All but about nbytes of the device's memory taken, in blocks, while the context is open."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    block = 1 << 36
    while block >= 2 * MB:
        while torch.cuda.mem_get_info()[0] >= nbytes + block:
            try:
                held.append(torch.empty(block, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                break
        block //= 2
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
        hp.upload_workload(wl)
        hp.full_pass()
        got = hp.download()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
