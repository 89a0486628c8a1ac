"""Plans in which a query is in several chunks (of one window here, so that it
does not matter which chunk's result is kept): every list of queries has room
for all of them."""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import rho_with_ties, small_site

pytestmark = pytest.mark.gpu


# rows, queries a chunk, step from chunk to chunk, listed neighbours: windows searched by a warp, by blocks, and 16
# queries at a time, with most lists too short to hold a higher rho
@pytest.mark.parametrize("n,nq,step,knn", [(500, 40, 8, 1), (1500, 40, 8, 1), (1500, 200, 25, 1), (2500, 300, 50, 30), (4800, 60, 10, 2)])
def test_queries_in_several_chunks(gpu, n, nq, step, knn):
    F, one, _ = small_site(n=n, d=12, n_chunks=1, seed=n, n_dup=10)
    q0 = np.arange(0, n - nq + 1, step)
    q0 = np.append(q0, n - nq) if q0[-1] != n - nq else q0
    c = len(q0)
    many = dict(one, q0=q0.astype(np.int32), nq=np.full(c, nq, np.int32), roff=np.arange(c + 1, dtype=np.int32),
                rs=np.zeros(c, np.int32), rn=np.full(c, n, np.int32))
    Fd = torch.from_numpy(F).to(gpu)
    P, Q = irc.Plan(one), irc.Plan(many)
    for mode in ("exact", "ref", "bf16"):
        a, b = irc.site_knn(P, Fd, knn, mode), irc.site_knn(Q, Fd, knn, mode)
        assert torch.equal(a["miKnn"], b["miKnn"]) and torch.equal(a["vrKnn"], b["vrKnn"]), mode
    R = rho_with_ties(n, 5)
    ex = irc.site_knn(P, Fd, knn, "exact")
    nn, d2 = O.exact_delta_f32(F, R, one)
    want = (np.sqrt(np.abs(d2)).astype(np.float32) * R).astype(np.float32)
    Rd = torch.from_numpy(R).to(gpu)
    for _ in range(2):
        delta, nneigh = irc.site_delta(Q, Fd, Rd, "exact", knn=knn, miKnn=ex["miKnn"], d2Knn=ex["d2Knn"])
        assert np.array_equal(nneigh.cpu().numpy(), nn)
        assert np.array_equal(delta.cpu().numpy().view(np.int32), want.view(np.int32))
    a, b = irc.site_delta(P, Fd, Rd, "ref", 512), irc.site_delta(Q, Fd, Rd, "ref", 512)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
