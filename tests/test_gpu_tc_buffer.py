"""The plan's tensor-core buffer keeps its size, and with it its place, over
layouts, unit widths and forms: a captured graph that uses it stays valid."""
import pytest
import torch

from ironclust_gb300 import _lib, irc
from tests.cases import small_site

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,chunks", [(20000, 24, 1), (9000, 33, 90), (400, 58, 20)])
def test_buffer_outlives_layout_changes(gpu, n, d, chunks):
    L = _lib.lib()
    F, plan, _ = small_site(n=n, d=d, n_chunks=chunks, seed=13)
    Fd = torch.from_numpy(F).to(gpu)
    P = irc.Plan(plan)
    size = L.irc_plan_tc_bytes(P.h, d)
    _lib.check(L.irc_plan_tc_units(P.h, 128), "irc_plan_tc_units")       # (no item is split at this width)
    Q = irc.Plan(plan)
    _lib.check(L.irc_plan_tc_units(Q.h, 128), "irc_plan_tc_units")
    irc.site_knn(Q, Fd, 30, "fp8")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):                                            # (an allocation would end the capture)
        got = irc.site_knn(Q, Fd, 30, "bf16")
    for slots in (1, 2, 4):
        for order in (0, 1):
            for width in (256, 128):
                _lib.check(L.irc_plan_tc_layout(Q.h, slots, order), "irc_plan_tc_layout")
                _lib.check(L.irc_plan_tc_units(Q.h, width), "irc_plan_tc_units")
                assert L.irc_plan_tc_bytes(Q.h, d) == size
                irc.site_knn(Q, Fd, 30, "bf16")
    irc.site_knn(P, Fd, 30, "bf16")
    for k in ("miKnn", "vrKnn"):
        got[k].zero_()
    g.replay()
    torch.cuda.synchronize()
    narrow = irc.site_knn(P, Fd, 30, "bf16")
    assert torch.equal(got["miKnn"], narrow["miKnn"]) and torch.equal(got["vrKnn"], narrow["vrKnn"])
