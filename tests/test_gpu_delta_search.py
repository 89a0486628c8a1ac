"""The drift-window search of the delta (irc_exact.cu) against the oracle, bit
for bit, at the edges of its split: windows searched by a warp, by a block, in
parts, and 16 queries at a time.

  peaks   rho of the kNN: a few density peaks without a listed neighbour
  ties    random rho with a tie group: most short lists hold no higher rho
  low     nearly every row has a higher rho than the queries that are searched
"""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import rho_with_ties, small_site

pytestmark = pytest.mark.gpu

# chunk sizes (a chunk's window is itself and its neighbours), D, listed neighbours
SHAPES = [
    ([17], 3, 1),
    ([511], 24, 2), ([512], 24, 2), ([513], 24, 2),            # a warp or a block per window
    ([2048], 12, 1), ([2049], 45, 1), ([4097], 24, 30),        # one part and two
    ([33000], 8, 30),                                          # the most parts
    ([63, 64, 65, 1, 900], 33, 1),                             # the fewest queries searched 16 at a time
    ([1500, 1200, 1700, 800], 59, 3),
]


@pytest.mark.parametrize("rho", ["peaks", "ties", "low"])
@pytest.mark.parametrize("sizes,d,knn", SHAPES)
def test_delta_search_equals_the_oracle(gpu, sizes, d, knn, rho):
    F, plan, _ = small_site(n=sum(sizes), d=d, seed=11 + d, sizes=sizes, n_dup=20)
    Fd = torch.from_numpy(F).to(gpu)
    P = irc.Plan(plan)
    ex = irc.site_knn(P, Fd, knn, "exact")
    R = rho_with_ties(F.shape[0], 5)
    if rho != "ties":
        R = ex["rho"].cpu().numpy().copy()
    if rho == "low":                                           # a few queries whose lists name row 1 only
        rng = np.random.default_rng(d)
        few = rng.choice(R.size, max(1, R.size // 200), replace=False)
        R[few] = np.float32(1e-6)
        R[0] = np.float32(0.0)
        ex["miKnn"][torch.from_numpy(few).to(gpu)] = 1
    delta, nneigh = irc.site_delta(P, Fd, torch.from_numpy(R).to(gpu), "exact", knn=knn, miKnn=ex["miKnn"], d2Knn=ex["d2Knn"])
    nn, d2 = O.exact_delta_f32(F, R, plan)
    assert np.array_equal(nneigh.cpu().numpy(), nn)
    want = np.sqrt(np.abs(d2)).astype(np.float32) * R[plan["q_base"]:plan["q_base"] + plan["n_out"]]
    assert np.array_equal(delta.cpu().numpy().view(np.int32), want.astype(np.float32).view(np.int32))
