"""nudim_diffusion2d and its scratch: a captured call allocates nothing, so its
graph may be instantiated and embedded like any other; calls on two streams of one
context, in flight together, do not share any."""
import ctypes

import numpy as np
import pytest

from gpu_util import rdtype, rel, to_dev

pytestmark = pytest.mark.gpu
KERNEL, MEM_ALLOC, MEM_FREE = 0, 10, 11  # CUgraphNodeType


def ok(status):
    assert status == 0, "CUDA error %d" % status


def volume(shape, seed):
    return 0.01 * np.random.default_rng(seed).standard_normal(shape)


def call(ctx, ng, d, prec, it, stream):
    ng.diffusion2d(ctx, d.data_ptr(), tuple(d.shape), d.shape[0], prec, 0.25, 0.005, it,
                   stream=stream)


@pytest.mark.parametrize("prec", [0, 1])
def test_captured_call_allocates_nothing(gpu_ctx, nudim_built, monkeypatch, prec):
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    p = ctypes.c_void_p
    v = volume((5, 70, 90), 1)
    d, st = to_dev(v, rdtype(prec)), torch.cuda.Stream()
    call(gpu_ctx, nudim_built, to_dev(v, rdtype(prec)), prec, 80, st.cuda_stream)
    torch.cuda.synchronize()
    graph = p()
    ok(cu.cuStreamBeginCapture_v2(p(st.cuda_stream), 1))  # thread-local
    call(gpu_ctx, nudim_built, d, prec, 80, st.cuda_stream)
    ok(cu.cuStreamEndCapture(p(st.cuda_stream), ctypes.byref(graph)))
    n = ctypes.c_size_t()
    ok(cu.cuGraphGetNodes(graph, None, ctypes.byref(n)))
    nodes = (p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)))
    types = []
    for x in nodes:
        t = ctypes.c_int()
        ok(cu.cuGraphNodeGetType(p(x), ctypes.byref(t)))
        types.append(t.value)
    assert KERNEL in types and MEM_ALLOC not in types and MEM_FREE not in types
    # two instances of it at once, and the calls that they stand for
    execs = [p(), p()]
    for e in execs:
        ok(cu.cuGraphInstantiateWithFlags(ctypes.byref(e), graph, ctypes.c_ulonglong(0)))
    for e in execs:
        ok(cu.cuGraphLaunch(e, p(st.cuda_stream)))
    torch.cuda.synchronize()
    eager = to_dev(v, rdtype(prec))
    for _ in execs:
        call(gpu_ctx, nudim_built, eager, prec, 80, None)
    torch.cuda.synchronize()
    got, want = d.cpu().numpy(), eager.cpu().numpy()
    if prec == 0:
        assert np.array_equal(got, want)
    assert rel(got, want) < 1e-5
    monkeypatch.setenv("NUDIM_DIFFUSION", "tables" if prec == 0 else "pairs")
    plain = to_dev(v, rdtype(prec))
    for _ in execs:
        call(gpu_ctx, nudim_built, plain, prec, 80, None)
    torch.cuda.synchronize()
    assert np.array_equal(got, plain.cpu().numpy())
    for e in execs:
        ok(cu.cuGraphExecDestroy(e))
    ok(cu.cuGraphDestroy(graph))


@pytest.mark.parametrize("prec", [0, 1])
def test_calls_on_two_streams(gpu_ctx, nudim_built, prec):
    import torch
    vs = [volume((6, 120, 100), 2), volume((9, 64, 200), 3)]
    want = []
    for v in vs:
        d = to_dev(v, rdtype(prec))
        for _ in range(8):
            call(gpu_ctx, nudim_built, d, prec, 40, None)
        torch.cuda.synchronize()
        want.append(d.cpu().numpy())
    ds, sts = [to_dev(v, rdtype(prec)) for v in vs], [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(8):
        for d, st in zip(ds, sts):
            call(gpu_ctx, nudim_built, d, prec, 40, st.cuda_stream)
    torch.cuda.synchronize()
    for d, w in zip(ds, want):
        assert np.array_equal(d.cpu().numpy(), w)
