"""Captured calls of the plain forms: graphs without allocations, which can be
instantiated more than once, also when the first call of a process is captured."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

from ironclust_gb300 import _lib, irc
from tests.cases import small_site

pytestmark = pytest.mark.gpu

MEM_ALLOC, MEM_FREE = 10, 11                                  # CU_GRAPH_NODE_TYPE_MEM_ALLOC, _MEM_FREE


def ok(rc):
    assert rc == 0, rc


def record(cu, stream, call):
    """The graph of the launches that call() makes on the stream (global capture mode)."""
    h, g = C.c_void_p(stream.cuda_stream), C.c_void_p()
    ok(cu.cuStreamBeginCapture_v2(h, 0))
    call()
    ok(cu.cuStreamEndCapture(h, C.byref(g)))
    return g


def node_types(cu, g):
    n = C.c_size_t()
    ok(cu.cuGraphGetNodes(g, None, C.byref(n)))
    nodes, t = (C.c_void_p * n.value)(), C.c_int()
    ok(cu.cuGraphGetNodes(g, nodes, C.byref(n)))
    out = []
    for x in nodes:
        ok(cu.cuGraphNodeGetType(C.c_void_p(x), C.byref(t)))
        out.append(t.value)
    return out


def run(mode, graphs):
    cu = C.CDLL("libcuda.so.1")
    dev = torch.device("cuda:0")
    F, plan, _ = small_site(n=7600, d=24, n_chunks=5, seed=7)
    Fd = torch.from_numpy(F).to(dev)
    P, L = irc.Plan(plan), _lib.lib()
    n = P.n_out
    vr, de = (torch.zeros(n, device=dev) for _ in range(2))
    rho = torch.rand(n, device=dev)
    mi, nn = torch.zeros((n, 30), dtype=torch.int32, device=dev), torch.zeros(n, dtype=torch.int32, device=dev)
    d2 = torch.zeros((n, 30), device=dev)
    s = torch.cuda.Stream()
    st, p = C.c_void_p(s.cuda_stream), irc._p

    def call():
        m = _lib.MODES[mode]
        _lib.check(L.irc_site_knn(P.h, p(Fd), 24, 30, 1024, m, p(vr), None, p(mi), p(d2) if mode == "exact" else None, st), "knn")
        if mode == "ref":
            _lib.check(L.irc_site_delta(P.h, p(Fd), 24, p(rho), 512, m, 30, None, None, p(de), p(nn), st), "delta")

    torch.cuda.synchronize()
    for _ in range(graphs):
        g = record(cu, s, call)
        types = node_types(cu, g)
        assert MEM_ALLOC not in types and MEM_FREE not in types
        execs = [C.c_void_p(), C.c_void_p()]
        for e in execs:
            ok(cu.cuGraphInstantiateWithFlags(C.byref(e), g, C.c_ulonglong(0)))
        got = []
        for e in execs:
            for t in (vr, de, mi, nn, d2):
                t.zero_()
            torch.cuda.synchronize()
            ok(cu.cuGraphLaunch(e, st))
            s.synchronize()
            got.append([t.clone() for t in (vr, mi, d2, de, nn)])
            ok(cu.cuGraphExecDestroy(e))
        ok(cu.cuGraphDestroy(g))
        want = irc.site_knn(P, Fd, 30, mode)
        dw = irc.site_delta(P, Fd, rho, "ref", 512) if mode == "ref" else (de * 0, nn * 0)
        for o in got:
            assert torch.equal(o[0], want["vrKnn"]) and torch.equal(o[1], want["miKnn"])
            assert torch.equal(o[3], dw[0]) and torch.equal(o[4], dw[1])


@pytest.mark.parametrize("mode", ["ref", "exact"])
def test_captured_calls_hold_no_allocations(gpu, mode):
    run(mode, 10)                                             # (more captured calls than a plan keeps memory for)


@pytest.mark.parametrize("mode", ["ref", "exact"])
def test_the_first_call_of_a_process_is_captured(gpu, mode):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = "import tests.test_gpu_graph_memory as t; t.run(%r, 1)" % mode
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
