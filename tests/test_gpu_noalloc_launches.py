"""gz_density_sums_noalloc promises a caller without free device memory that its first call loads everything: so the
kernels of a call must not depend on the number of particles. A captured call of each size shows which they are; its
replay gives the sums of the plain call."""
import ctypes as C

import numpy as np
import pytest

from gizmo_b200 import abi, ics

pytestmark = pytest.mark.gpu


def _inputs(n):
    import torch

    wl = ics.plummer_mix(41, seed=6, n_spheres=12)
    f = {k: torch.as_tensor(np.ascontiguousarray(getattr(wl, k)[:n]), device="cuda") for k in ("pos", "vel", "mass", "h")}
    f["acc"] = torch.zeros(n, 14, dtype=torch.float64, device="cuda")
    f["pv"] = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    return wl.params, f


def _call(params, f):
    import torch

    rc = abi.load_library().gz_density_sums_noalloc(
        C.byref(params), f["mass"].shape[0], *(f[k].data_ptr() for k in ("pos", "vel", "mass", "h", "acc", "pv")),
        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == abi.OK


def _kernels(graph):
    """Names of the kernels of a captured graph, all of whose nodes are kernels."""
    from cuda.bindings import driver as D

    raw = D.CUgraph(int(graph.raw_cuda_graph()))
    count = D.cuGraphGetNodes(raw, 0)[2]
    names = []
    for node in D.cuGraphGetNodes(raw, count)[1]:
        assert D.cuGraphNodeGetType(node)[1] == D.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL
        names.append(D.cuFuncGetName(D.cuGraphKernelNodeGetParams(node)[1].func)[1])
    return names


def test_every_call_launches_the_same_kernels():
    import torch

    kernels = {}
    for n in (1, 33, 1000, 4097, 20001, 65536):
        params, f = _inputs(n)
        _call(params, f)
        torch.cuda.synchronize()
        plain = f["acc"].clone()
        f["acc"].zero_()
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            _call(params, f)
        kernels[n] = _kernels(g)
        assert not f["acc"].any()  # captured, not run
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(f["acc"], plain)
    assert len(kernels[1]) >= 3
    for n in kernels:
        assert kernels[n] == kernels[1], n


def test_overlapping_calls_stay_inside_their_arrays():
    """Calls that overlap on the GPU have undefined results, and nothing more: a small set's outputs lie between
    guards while calls of a large one rewrite the scratch under it, and a call by itself is right afterwards."""
    import torch

    n, guard = 1000, 70000
    params, large = _inputs(65536)
    _, small = _inputs(n)
    _call(params, small)
    torch.cuda.synchronize()
    want, want_pv = small["acc"].clone(), small["pv"].clone()
    acc = torch.full((n + 2 * guard, 14), -7.0, dtype=torch.float64, device="cuda")
    pv = torch.full((n + 2 * guard, 3), -7.0, dtype=torch.float64, device="cuda")
    inside = dict(small, acc=acc[guard:guard + n], pv=pv[guard:guard + n])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(200):
        for s, f in zip(streams, (large, inside)):
            with torch.cuda.stream(s):
                _call(params, f)
    torch.cuda.synchronize()
    for t in (acc, pv):
        assert (t[:guard] == -7.0).all() and (t[guard + n:] == -7.0).all()
    _call(params, inside)
    torch.cuda.synchronize()
    assert torch.equal(inside["acc"], want) and torch.equal(inside["pv"], want_pv)
