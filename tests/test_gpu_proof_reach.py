"""What the proven search of the plain forms leaves to the plain kernels
(irc_plan_search_counts), and its results against theirs: a plan that names a
query twice is served by the plain kernels alone."""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc, synth

pytestmark = pytest.mark.gpu


def plain_plan(plan):
    """The plan, and its first query once more: searched by the plain kernels."""
    r = int(plan["roff"][1])
    i32 = lambda a, *more: np.concatenate([a, *more]).astype(np.int32)
    return dict(plan, q0=i32(plan["q0"], plan["q0"][:1]), nq=i32(plan["nq"], [1]), roff=i32(plan["roff"], [plan["roff"][-1] + r]),
                rs=i32(plan["rs"], plan["rs"][:r]), rn=i32(plan["rn"], plan["rn"][:r]))


def check(gpu, F, plan, knn=30, nT=1024):
    """(tiles left by EXACT, by REF, queries left by the REF delta), outputs equal to the plain kernels'."""
    Fd = torch.from_numpy(np.ascontiguousarray(F)).to(gpu)
    P, Q = irc.Plan(plan), irc.Plan(plain_plan(plan))
    left = []
    for mode in ("exact", "ref"):
        a, b = irc.site_knn(P, Fd, knn, mode, nT), irc.site_knn(Q, Fd, knn, mode, nT)
        for k in ("miKnn", "vrKnn", "d2Knn"):
            if a[k] is not None:
                assert torch.equal(a[k].view(torch.int32), b[k].view(torch.int32)), (mode, k)
        c, plain = P.search_counts(), Q.search_counts()
        assert c["searches"] == 1 and plain["searches"] == 0   # (the control is the plain kernels)
        assert c["scans"] <= plain["scans"]                    # (rows so far out that all their distances round to the same)
        left.append(c["tiles"])
    rho = torch.nan_to_num(b["rho"])
    a, b = irc.site_delta(P, Fd, rho, "ref", 512), irc.site_delta(Q, Fd, rho, "ref", 512)
    assert torch.equal(a[0].view(torch.int32), b[0].view(torch.int32)) and torch.equal(a[1], b[1])
    c = P.search_counts()
    assert Q.search_counts()["deltas"] == 0
    return (*left, c["windows"] if c["deltas"] else None)      # (None: too small for the search)


@pytest.mark.parametrize("size", [3e3, 1e5, 1e9, 1e30, np.inf, np.nan])
@pytest.mark.parametrize("n,d,chunks", [(7301, 24, 1), (10000, 33, 4)])
def test_far_rows_do_not_spoil_the_proof(gpu, n, d, chunks, size):
    """Five rows far out (some sampled for the centre) cost their own tiles, no others."""
    s = synth.make_site(n, d, 12, chunks, 17)
    F = s["F"].copy()
    rng = np.random.default_rng(3)
    F[rng.choice(n, 5, replace=False)] = (size * rng.normal(1.0, 0.3, (5, d))).astype(np.float32)
    exact, ref, windows = check(gpu, F, synth.site_plan(s))
    assert exact <= 5 and ref <= 5 and windows <= n // 50


@pytest.mark.parametrize("shift", [0.0, 1e4])
def test_an_offset_does_not_either(gpu, shift):
    s = synth.make_site(8000, 24, 12, 3, 19)
    exact, ref, windows = check(gpu, (s["F"] + np.float32(shift)).astype(np.float32), synth.site_plan(s))
    assert exact == 0 and ref == 0 and windows <= 160


def spread_site(n, d, chunks, spread, seed=23):
    """A site whose units lie `spread` (in units of a typical noise) apart."""
    s = synth.make_site(n, d, 12, chunks, seed)
    rng = np.random.default_rng(seed)
    F, lab = s["F"].astype(np.float64), s["labels"]
    m = lab >= 0
    c = rng.normal(0.0, 1.0, (12, d))
    F[m] += c[lab[m]] * spread
    F[~m] = rng.uniform(F[m].min(0), F[m].max(0), ((~m).sum(), d))
    return F.astype(np.float32), synth.site_plan(s)


# the windows of open queries are read again: a few queries, most of them, all; one part and several, runs of a few
# rows, fewer queries than a group, D to the operand row's limit, knn 1 and 32, bins that runs do and do not divide
@pytest.mark.parametrize("n,d,chunks,spread,knn,nT", [
    (2600, 33, 1, 30, 30, 1024), (7301, 24, 1, 40, 30, 1024), (7301, 24, 1, 100, 30, 1000), (9000, 33, 300, 80, 30, 1024),
    (20011, 24, 600, 300, 32, 1024), (7205, 58, 2, 200, 1, 1024), (12000, 3, 5, 1000, 30, 512), (30011, 24, 2, 60, 17, 256),
    (40000, 24, 1, 100, 30, 1024)])
def test_open_queries_get_a_second_look(gpu, n, d, chunks, spread, knn, nT):
    F, plan = spread_site(n, d, chunks, spread)
    exact, ref, _ = check(gpu, F, plan, knn, nT)
    assert exact == 0 and ref == 0


@pytest.mark.parametrize("chunks", [1, 40, 400])
def test_windows_with_fewer_rows_than_neighbours(gpu, chunks):
    """Chunks that are their own windows, of 1 to 60 rows, beside wide ones."""
    rng = np.random.default_rng(chunks)
    sizes = np.concatenate([rng.integers(1, 61, chunks), [6000, 3000]]).astype(np.int32)
    q0 = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    n = int(sizes.sum())
    plan = dict(q0=q0, nq=sizes, roff=np.arange(len(sizes) + 1, dtype=np.int32), rs=q0, rn=sizes, q_base=0, n_out=n, n_f=n)
    F = synth.make_site(n, 24, 12, 1, 5)["F"]
    F[100:140] = F[100]
    check(gpu, F, plan)
    check(gpu, F, plan, 32, 96)


def test_copies_and_ties(gpu):
    """More copies than a list holds, and more equal distances than are collected, go to the plain kernels."""
    s = synth.make_site(8000, 6, 12, 2, 29)
    F = np.round(s["F"])                                       # whole numbers: equal distances everywhere
    F[1000:1400] = F[1000]
    exact, ref, _ = check(gpu, F, synth.site_plan(s))
    assert exact > 0 and ref > 0
