"""The plain forms through the proven tensor-core search (irc_cert.cu) against
the oracle: REF kNN and delta, EXACT kNN, bit for bit, on sites large enough
for the search to be taken and on data that must fall back to the
plain kernels in part or in whole.

  dup      exact copies of spikes: zero distances, equal distances
  outlier  a few spikes at 1e6 and one that is not finite: the operands' scale
           and centre must not break the proof for the others
  shift    every feature offset by 1e4: half-precision operands are centred
  coarse   clusters far apart and tiny inside: the proof fails everywhere
"""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc, synth
from ironclust_gb300.drift import build_plan
from oracle import oracle as O
from tests.cases import rho_with_ties, small_site

pytestmark = pytest.mark.gpu


def bits(a):
    a = a.detach().cpu().numpy() if isinstance(a, torch.Tensor) else np.ascontiguousarray(a)
    return a.view(np.int32) if a.dtype == np.float32 else a


def make(kind, n, d, chunks, seed, secondary=False):
    F, plan, _ = small_site(n=n, d=d, n_chunks=chunks, seed=seed, n_dup=200 if kind == "dup" else 0, secondary=secondary)
    rng = np.random.default_rng(seed)
    if kind == "outlier":
        F[rng.choice(F.shape[0], 5, replace=False)] = rng.normal(0, 1e6, (5, d)).astype(np.float32)
        F[17, 0] = np.nan
        F[18, d - 1] = np.inf
    if kind == "shift":
        F = (F + np.float32(1e4)).astype(np.float32)
    if kind == "coarse":
        F = (np.round(F / 50.0) * 1e4 + 1e-2 * rng.standard_normal(F.shape)).astype(np.float32)
    return np.ascontiguousarray(F), plan


def ref_oracle(F, plan, knn, nT):
    n = plan["n_out"]
    vr, mi = np.zeros(n, np.float32), np.zeros((n, knn), np.int32)
    for i in range(len(plan["q0"])):
        r0, r1 = plan["roff"][i], plan["roff"][i + 1]
        q0, nq = int(plan["q0"][i]), int(plan["nq"][i])
        D, I = O.search_min_drift(F, plan["rs"][r0:r1], plan["rn"][r0:r1], [F.shape[1], F.shape[0], int(r1 - r0), q0, nq], nT)
        o = q0 - plan["q_base"]
        vr[o:o + nq], mi[o:o + nq] = O.post_sort_knn(D, I, knn)
    return vr, mi


def ref_delta_oracle(F, R, plan, nT):
    n = plan["n_out"]
    de, nn = np.zeros(n, np.float32), np.zeros(n, np.int32)
    for i in range(len(plan["q0"])):
        r0, r1 = plan["roff"][i], plan["roff"][i + 1]
        q0, nq = int(plan["q0"][i]), int(plan["nq"][i])
        D, I = O.search_delta_drift(F, R, plan["rs"][r0:r1], plan["rn"][r0:r1],
                                    [F.shape[1], F.shape[0], int(r1 - r0), q0, nq], nT)
        o = q0 - plan["q_base"]
        v, m = O.post_min(D, I)
        de[o:o + nq], nn[o:o + nq] = v * R[q0:q0 + nq], m
    return de, nn


# n, d, chunks, secondary copies, knn, REF bins: tiles and units with remainders, one chunk, D to the operand
# row's limit (58; 59 goes to the plain kernels), knn 1 and 32, bins that the runs do and do not divide
SHAPES = [
    ("plain", 7600, 24, 5, False, 30, 1024),
    ("dup", 6900, 33, 4, True, 30, 1024),
    ("plain", 8001, 3, 1, False, 1, 1024),
    ("outlier", 7301, 18, 1, False, 30, 1000),
    ("shift", 7299, 45, 3, False, 32, 1024),
    ("coarse", 7200, 12, 2, False, 30, 512),
    ("dup", 7200, 55, 1, False, 17, 256),
    ("plain", 7200, 58, 1, False, 30, 1024),
    ("plain", 7200, 59, 1, False, 30, 1024),
    ("plain", 20011, 24, 600, False, 30, 1024),
    # the smallest sites of the search: fewer queries than a tile's columns, windows of a few hundred rows
    ("plain", 905, 25, 1, False, 30, 1024), ("dup", 1100, 45, 2, True, 32, 1000), ("shift", 2101, 24, 3, False, 30, 512),
    ("outlier", 2405, 9, 1, False, 30, 1024), ("coarse", 3001, 12, 40, False, 5, 1024), ("plain", 4003, 6, 200, False, 30, 1024),
]


@pytest.mark.parametrize("kind,n,d,chunks,secondary,knn,nT", SHAPES)
def test_plain_forms_equal_the_oracle(gpu, kind, n, d, chunks, secondary, knn, nT):
    F, plan = make(kind, n, d, chunks, 31 + d, secondary)
    Fd = torch.from_numpy(F).to(gpu)
    P = irc.Plan(plan)
    out = irc.site_knn(P, Fd, knn, "ref", nT)
    vr, mi = ref_oracle(F, plan, knn, nT)
    assert np.array_equal(out["miKnn"].cpu().numpy(), mi)
    assert np.array_equal(bits(out["vrKnn"]), bits(vr))
    R = rho_with_ties(F.shape[0], 5)
    de, nn = ref_delta_oracle(F, R, plan, nT)
    delta, nneigh = irc.site_delta(P, Fd, torch.from_numpy(R).to(gpu), "ref", nT)
    assert np.array_equal(nneigh.cpu().numpy(), nn)
    assert np.array_equal(bits(delta), bits(de))
    if kind == "outlier":
        return                                           # the EXACT oracle has no rule for rows that are not finite
    ex = irc.site_knn(P, Fd, knn, "exact")
    idx, d2 = O.exact_knn_f32(F, plan, knn)
    assert np.array_equal(ex["miKnn"].cpu().numpy(), idx)
    assert np.array_equal(bits(ex["d2Knn"]), bits(d2))


def test_under_capture_and_on_two_streams(gpu):
    """The working memory is stream-ordered: a captured call replays, and calls
    of one plan on two streams do not share it."""
    F, plan, _ = small_site(n=7600, d=24, n_chunks=5, seed=7)
    F2 = np.ascontiguousarray(F[:, ::-1])
    P = irc.Plan(plan)
    a, b = torch.from_numpy(F).to(gpu), torch.from_numpy(F2).to(gpu)
    want = {k: [irc.site_knn(P, x, 30, k) for x in (a, b)] for k in ("ref", "exact")}
    torch.cuda.synchronize()
    for mode in ("ref", "exact"):
        x = a.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = irc.site_knn(P, x, 30, mode)
        for src, w in ((b, want[mode][1]), (a, want[mode][0])):
            x.copy_(src)
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(got["miKnn"], w["miKnn"]) and torch.equal(got["vrKnn"], w["vrKnn"]), mode
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for s in (s1, s2):
        s.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(5):
        with torch.cuda.stream(s1):
            outs.append((0, irc.site_knn(P, a, 30, "ref")))
        with torch.cuda.stream(s2):
            outs.append((1, irc.site_knn(P, b, 30, "ref")))
    torch.cuda.synchronize()
    for i, o in outs:
        assert torch.equal(o["miKnn"], want["ref"][i]["miKnn"]) and torch.equal(o["vrKnn"], want["ref"][i]["vrKnn"])
