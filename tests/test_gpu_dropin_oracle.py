"""The drop-in kernels against the C oracle, bit for bit, at the edges of their
tiles: 16- and 8-query CTAs, 256-bin turns, bins with and without candidates,
feature counts with every load width and both shared-memory layouts (even, odd,
the largest), candidates in one and in many cluster slices, ties, exact copies.
"""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import rho_with_ties, small_site

pytestmark = pytest.mark.gpu


def bits(a):
    a = a.detach().cpu().numpy() if isinstance(a, torch.Tensor) else np.ascontiguousarray(a)
    return a.view(np.int32) if a.dtype in (np.float32, np.uint32) else a


def same(a, b):
    return np.array_equal(bits(a), bits(b))


def features(rng, n, nC):
    F = rng.normal(0, 2, (n, nC)).astype(np.float32)
    k = min(n // 3, 40)
    F[n - k:] = F[:k]                                     # exact copies: zero and equal distances
    return F


@pytest.mark.parametrize("n,d,chunks,nTk,nTd,secondary", [
    (2003, 24, 4, 1024, 512, False), (1501, 33, 3, 1000, 500, True), (901, 1, 1, 257, 255, False),
    (700, 64, 2, 512, 1024, False), (333, 18, 1, 33, 7, False)])
def test_search_drift(gpu, n, d, chunks, nTk, nTd, secondary):
    F, plan, _ = small_site(n=n, d=d, n_chunks=chunks, seed=n, n_dup=60, secondary=secondary)
    R = rho_with_ties(F.shape[0], 3)
    Fd, Rd = torch.from_numpy(F).to(gpu), torch.from_numpy(R).to(gpu)
    for i in range(len(plan["q0"])):
        r0, r1 = plan["roff"][i], plan["roff"][i + 1]
        rs, rn = np.ascontiguousarray(plan["rs"][r0:r1]), np.ascontiguousarray(plan["rn"][r0:r1])
        vn = [d, F.shape[0], int(r1 - r0), int(plan["q0"][i]), int(plan["nq"][i])]
        t = [torch.from_numpy(x).to(gpu) for x in (rs, rn)]
        D, I = irc.search_min_drift(Fd, *t, vn, nTk)
        Do, Io = O.search_min_drift(F, rs, rn, vn, nTk)
        assert same(D, Do) and same(I, Io), i
        D, I = irc.search_delta_drift(Fd, Rd, *t, vn, nTd)
        Do, Io = O.search_delta_drift(F, R, rs, rn, vn, nTd)
        assert same(D, Do) and same(I, Io), i


@pytest.mark.parametrize("nB,nA,nC,knn,nT", [
    (1500, 200, 33, 30, 512), (300, 77, 24, 30, 512), (40, 17, 18, 40, 512), (5000, 33, 60, 30, 512),
    (2000, 2500, 30, 30, 512), (3000, 9, 64, 31, 1024), (700, 65, 1, 5, 256), (900, 2433, 64, 30, 1024)])
def test_binned_knn(gpu, nB, nA, nC, knn, nT):
    rng = np.random.default_rng(nB + nA)
    B = features(rng, nB, nC)
    A = np.concatenate([B[: nA // 2], features(rng, nA - nA // 2, nC)])[:nA]
    Bd, Ad = torch.from_numpy(B).to(gpu), torch.from_numpy(np.ascontiguousarray(A)).to(gpu)
    K, I = irc.cuda_knn_index(Bd, Ad, knn, nT)
    Ko, Io = O.cuda_knn_index(B, A, knn, nT)
    assert same(K, Ko) and same(I, Io)
    assert same(irc.cuda_knn_kth(Bd, Ad, knn, nT), O.cuda_knn(B, A, knn, nT))
    K, I = irc.cuda_knn_full(Bd, Ad, knn, nT)
    Ko, Io = O.cuda_knn_full(B, A, knn, nT)
    assert same(K, Ko) and same(I, Io)
    IB = rng.integers(1, nB + 1, nB // 2 + 1).astype(np.int32)
    K, I = irc.cuda_knn_ib(Bd, Ad, IB, knn, nT)
    Ko, Io = O.cuda_knn_ib(B, A, IB, knn, nT)
    assert same(K, Ko) and same(I, Io)


@pytest.mark.parametrize("nB,nA,nC", [(1500, 200, 33), (100, 300, 24), (3000, 16, 45), (20000, 130, 18), (9000, 5000, 2),
                                      (4100, 33, 64), (1, 1, 5)])
def test_delta_knn(gpu, nB, nA, nC):
    rng = np.random.default_rng(nB * 3 + nA)
    B, A = features(rng, nB, nC), features(rng, nA, nC)
    RB, RA = rho_with_ties(nB, 1), rho_with_ties(nA, 2)
    RA[0] = 2.0                                           # nothing above it
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(gpu)
    D, N = irc.cuda_delta_knn(t(B), t(A), t(RB), t(RA))
    Do, No = O.cuda_delta_knn(B, A, RB, RA)
    assert same(D, Do) and same(N, No)


@pytest.mark.parametrize("n12,n1,nC,sites,shift", [(1500, 300, 33, 3, 0), (700, 700, 24, 40, 0), (2000, 17, 45, 1, 0),
                                                   (4000, 31, 18, 64, 0), (3001, 33, 16, 5, 1), (50, 50, 64, 3, 0)])
def test_drift_window(gpu, n12, n1, nC, sites, shift):
    rng = np.random.default_rng(n12 + n1)
    f1 = features(rng, n12, nC)
    f2 = (f1 + rng.normal(0, 0.5, (n12, nC))).astype(np.float32)
    s1 = rng.integers(1, sites + 1, n12).astype(np.int32)
    s2 = rng.integers(0, sites + 1, n12).astype(np.int32)
    rho = rho_with_ties(n12, 9)
    dc2 = float(np.float32(1.7 * nC))

    def t(x):                                             # `shift` floats off a 16-byte boundary
        x = torch.from_numpy(np.ascontiguousarray(x))
        b = torch.empty(x.numel() + shift, dtype=x.dtype, device=gpu)
        b[shift:].copy_(x.reshape(-1))
        return b[shift:].view(x.shape)
    site = torch.from_numpy(np.concatenate([s1, s2])).to(gpu)
    got = irc.rho_drift(site, t(f1), t(f2), n1, dc2)
    assert same(got, O.rho_drift(np.stack([s1, s2], 1), f1, f2, n1, dc2))
    de, nn = irc.delta_drift(site, t(f1), t(f2), torch.from_numpy(rho).to(gpu), n1, dc2)
    do, no = O.delta_drift(np.stack([s1, s2], 1), f1, f2, rho, n1, dc2)
    assert same(de, do) and same(nn, no)
