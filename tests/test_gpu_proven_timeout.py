"""REF and EXACT calls of the proven search when the filter's waits give up: every
tile (every query of the delta) is searched by the plain kernels, and the outputs
are theirs, also with items split over their candidates."""
import pytest
import torch

from ironclust_gb300 import _lib, irc, synth
from tests.test_gpu_proof_reach import plain_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,chunks", [(7600, 24, 5), (20000, 24, 1), (9000, 18, 400)])
def test_waits_that_give_up_leave_every_tile(gpu, n, d, chunks):
    L = _lib.lib()
    s = synth.make_site(n, d, 12, chunks, 5)
    plan, F = synth.site_plan(s), torch.from_numpy(s["F"]).to(gpu)
    P, Q = irc.Plan(plan), irc.Plan(plain_plan(plan))
    tiles = int(sum(-(-int(x) // 16) for x in plan["nq"]))
    rho = irc.site_knn(Q, F, 30, "ref")["rho"]
    want = {m: irc.site_knn(Q, F, 30, m) for m in ("ref", "exact")}
    dwant = irc.site_delta(Q, F, rho, "ref", 512)
    _lib.check(L.irc_set_wait_limit(2), "irc_set_wait_limit")
    try:
        for mode in ("ref", "exact"):
            got = irc.site_knn(P, F, 30, mode)
            c = P.search_counts()
            assert c["searches"] == 1 and c["tiles"] == tiles
            for k in ("miKnn", "vrKnn", "d2Knn"):
                if got[k] is not None:
                    assert torch.equal(got[k].view(torch.int32), want[mode][k].view(torch.int32)), (mode, k)
        got = irc.site_delta(P, F, rho, "ref", 512)
        c = P.search_counts()
        assert c["windows"] == (n if c["deltas"] else 0)
        assert torch.equal(got[0].view(torch.int32), dwant[0].view(torch.int32)) and torch.equal(got[1], dwant[1])
    finally:
        _lib.check(L.irc_set_wait_limit(0), "irc_set_wait_limit")
    irc.site_knn(P, F, 30, "exact")
    assert P.search_counts()["tiles"] == 0
