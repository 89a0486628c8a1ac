"""The list delta on lists that end early: entries behind a list's end, and
entries that name no row, are not used as row numbers."""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import rho_with_ties, small_site

pytestmark = pytest.mark.gpu

BIG = 2**31 - 1
# (index, squared distance) behind the end: MATLAB-style padding, the library's, indices outside F
TAILS = [(0, np.inf), (0, 3.402e38), (-5, np.nan), (BIG, np.inf), (-BIG, 3.402e38), (BIG, 1.0), (0, 1.0), (-BIG, 0.5)]


@pytest.mark.parametrize("knn", [1, 4, 7, 30])
@pytest.mark.parametrize("tail", TAILS)
def test_list_tails(gpu, knn, tail):
    F, plan, _ = small_site(n=1501, d=12, n_chunks=3, seed=23, n_dup=20)
    n = F.shape[0]
    idx, d2 = O.exact_knn_f32(F, plan, knn)
    rng = np.random.default_rng(knn)
    end = rng.integers(0, knn + 1, n)                          # the list's length, 0 .. knn
    cut = np.arange(knn)[None] >= end[:, None]
    idx, d2 = np.where(cut, tail[0], idx).astype(np.int32), np.where(cut, tail[1], d2).astype(np.float32)
    R = rho_with_ties(n, 5)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(gpu)
    delta, nneigh = irc.site_delta(irc.Plan(plan), dev(F), dev(R), "exact", knn=knn, miKnn=dev(idx), d2Knn=dev(d2))
    nn, dd = O.exact_delta_f32(F, R, plan)
    assert np.array_equal(nneigh.cpu().numpy(), nn)
    want = (np.sqrt(np.abs(dd)).astype(np.float32) * R).astype(np.float32)
    assert np.array_equal(delta.cpu().numpy().view(np.int32), want.view(np.int32))
