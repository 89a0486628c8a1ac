"""The drop-in kernels on both sides of the lines between their staged and their
direct forms, against the C oracle, bit for bit."""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import rho_with_ties
from tests.test_gpu_dropin_oracle import features, same

pytestmark = pytest.mark.gpu


# rows, features, runs, queries, bins
@pytest.mark.parametrize("n,d,runs,nA,nT", [
    (1000, 18, 1, 70, 512), (1000, 19, 1, 70, 512), (1000, 25, 3, 33, 512), (1000, 26, 3, 33, 512), (2048, 9, 1, 17, 512),
    (2049, 9, 1, 17, 512), (1024, 12, 1, 65, 1024), (1024, 12, 1, 64, 1024), (1025, 6, 1, 100, 1024), (300, 45, 3, 66, 1024),
    (300, 46, 3, 66, 1024), (5000, 12, 3, 4864, 1024), (5000, 13, 3, 4864, 1024), (5000, 6, 3, 4864, 512), (5, 64, 2, 3, 257),
    (1, 1, 1, 1, 1024)])
def test_search_forms(gpu, n, d, runs, nA, nT):
    rng = np.random.default_rng(n + d)
    F, R = features(rng, n, d), rho_with_ties(n, 3)
    cut = np.linspace(0, n, runs + 1).astype(np.int32)
    rs, rn = cut[:-1].copy(), np.diff(cut).astype(np.int32)
    vn = [d, n, runs, n - nA, nA]
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(gpu)
    D, I = irc.search_min_drift(t(F), t(rs), t(rn), vn, nT)
    Do, Io = O.search_min_drift(F, rs, rn, vn, nT)
    assert same(D, Do) and same(I, Io)
    D, I = irc.search_delta_drift(t(F), t(R), t(rs), t(rn), vn, nT)
    Do, Io = O.search_delta_drift(F, R, rs, rn, vn, nT)
    assert same(D, Do) and same(I, Io)


@pytest.mark.parametrize("nB,nA,nC", [(1024, 33, 30), (1025, 33, 30), (1500, 4864, 9), (1500, 4863, 9), (1500, 4864, 10), (127, 16, 64),
                                      (129, 4900, 1), (20000, 9800, 3)])
def test_delta_forms(gpu, nB, nA, nC):
    rng = np.random.default_rng(nB * 3 + nA)
    B, A = features(rng, nB, nC), features(rng, nA, nC)
    B[5], A[3] = np.nan, np.inf
    RB, RA = rho_with_ties(nB, 1), rho_with_ties(nA, 2)
    RA[0] = 2.0                                           # nothing above it
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(gpu)
    D, N = irc.cuda_delta_knn(t(B), t(A), t(RB), t(RA))
    Do, No = O.cuda_delta_knn(B, A, RB, RA)
    assert same(D, Do) and same(N, No)
