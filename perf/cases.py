"""The work whose speed this repository looks after: one pass of each public path, at sizes from a small site to a long recording.

Data are the seeded synthetic sites of ironclust_gb300.synth / .stream (Gaussian clusters with 5 % noise, drift as a random walk of the
chunk centres, every chunk linked to its 15 most similar within +-64), knn = 30.  The FP8 form is left out: its kNN recall is below the
bar of the path, so it is not used in earnest.
"""
import math

import numpy as np
import torch

from ironclust_gb300 import batch, irc, stream, synth

KNN = 30
LINKS = 15
SINGLE_INF = 3.402e38


def listed():
    return [
        # a small site of a short recording, with the copies that spikes of neighbouring sites leave on it: latency and launches count
        dict(name="site_bf16_small", kind="site", mode="bf16", n=3001, d=18, chunks=7, clusters=8, copies=1000),
        # one static site (no drift), the reference's plain single-chunk shape
        dict(name="site_bf16_static20k", kind="site", mode="bf16", n=20000, d=24, chunks=1, clusters=12, copies=0),
        # one drift site of a long recording: the headline shape of bench.py
        dict(name="site_bf16_drift400k", kind="site", mode="bf16", n=400000, d=33, chunks=200, clusters=16, copies=0),
        # the sites of a probe in one batch, ~20 spikes per site and chunk
        dict(name="probe_bf16", kind="probe", mode="bf16", sites=24, n=625000, chunks=1200),
        # the true kNN in plain FP32, a ragged drift site
        dict(name="site_exact_drift", kind="site", mode="exact", n=100003, d=33, chunks=50, clusters=16, copies=0),
        # the default mode, bit for bit the reference's binned search, with copies of neighbouring sites' spikes
        dict(name="site_ref_drift", kind="site", mode="ref", n=60001, d=24, chunks=30, clusters=12, copies=12001),
        # an unchanged irc2 host loop: one drift chunk through the two drop-in kernels
        dict(name="chunk_dropin", kind="chunk", n=30000, d=33, chunks=15, clusters=16),
        # an unchanged irc (v4) host loop: one drift chunk's kNN and delta through the wrappers
        dict(name="v4_knn_delta", kind="v4", n=15000, n_own=1507, d=30, clusters=12),
        # one window of the time-drift mode over the sites of a probe
        dict(name="v4_drift_window", kind="window", n=20011, n_own=2003, d=18, sites=64),
        # a site from features to clusters: kNN, rho, delta, sort, merge, propagation
        dict(name="site_to_clusters", kind="clusters", mode="bf16", n=100000, d=33, chunks=50, clusters=16),
        # the drift linkage of a whole recording
        dict(name="calc_drift", kind="linkage", n=1000000, sites=64, chunks=400, batch=15),
        # a recording larger than the working set, paged from pinned host memory as FP16
        dict(name="stream_fp16", kind="stream", mode="bf16", sites=16, n=800000, chunks=512, d=33),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["site"] * 5 + ["probe", "chunk", "v4", "window", "clusters", "linkage", "stream"])
    d = rng.choice([rng.randint(6, 45), 3 * rng.randint(3, 15)])
    clusters = rng.randint(4, 40)
    if kind in ("site", "clusters"):
        mode = rng.choice(["bf16", "bf16", "exact", "ref"]) if kind == "site" else "bf16"
        n = _log_int(rng, 500, 400000 if kind == "site" and mode == "bf16" else 100000)
        chunks = 1 if n <= 20000 and rng.random() < 0.3 else max(1, min(250, n // rng.randint(400, 2500)))
        c = dict(kind=kind, mode=mode, n=n, d=d, chunks=chunks, clusters=clusters)
        if kind == "site":
            c["copies"] = rng.choice([0, n // rng.randint(3, 9)]) if n <= 100000 else 0
        while _site_pairs(c) * d > 1.2e10 * 33 * (1.0 if mode == "bf16" else 0.25):
            c["chunks"] += 1
        return c
    if kind == "probe":
        sites = rng.randint(3, 24)
        return dict(kind=kind, mode="bf16", sites=sites, n=sites * _log_int(rng, 4000, 26000), chunks=rng.randint(300, 1200))
    if kind == "chunk":
        chunks = rng.randint(2, 15)
        return dict(kind=kind, n=chunks * rng.randint(100, 2000) + rng.randint(0, 50), d=d, chunks=chunks, clusters=clusters)
    if kind == "v4":
        n = _log_int(rng, 600, 20000)
        return dict(kind=kind, n=n, n_own=max(20, n // rng.randint(1, 15)), d=d, clusters=clusters)
    if kind == "window":
        n = _log_int(rng, 1000, 30000)
        return dict(kind=kind, n=n, n_own=max(20, n // rng.randint(3, 15)), d=3 * rng.randint(2, 9), sites=rng.randint(8, 128))
    if kind == "linkage":
        return dict(kind=kind, n=_log_int(rng, 20000, 1000000), sites=rng.randint(16, 128), chunks=rng.randint(40, 400), batch=LINKS)
    return dict(kind=kind, mode="bf16", sites=rng.randint(4, 16), n=_log_int(rng, 100000, 800000), chunks=rng.randint(300, 640), d=d)


# ---- what a user's program has in hand ---------------------------------------------------------------------------------------------

def _site(case, seed):
    """(F [nF, d], plan): the site's spikes, then the copies of neighbouring sites' spikes, each in time order."""
    n, d, copies = case["n"], case["d"], case.get("copies", 0)
    s = synth.make_site(n, d, case["clusters"], case["chunks"], seed)
    F, vd = s["F"], s["viDrift"]
    vl = np.ones(n, bool)
    if copies:
        r = np.random.default_rng(seed + 77)
        pick = np.sort(r.choice(n, size=copies, replace=False))
        F = np.concatenate([F, F[pick] + r.normal(0, 1.0, (copies, d)).astype(np.float32)])
        vd = np.concatenate([vd, vd[pick]])
        vl = np.concatenate([vl, np.zeros(copies, bool)])
    return np.ascontiguousarray(F, np.float32), synth.build_plan(vd, vl, s["mlDrift"])


def _probe(case, seed):
    r = np.random.default_rng(case["n"])                             # spike counts go with the case, spikes with the seed
    n = np.exp(r.normal(0.0, 1.0, case["sites"]))
    n = np.maximum((n * case["n"] / n.sum()).astype(np.int64), 500)
    dims = r.choice([18, 24, 33], size=case["sites"])
    return batch.SiteBatch(synth.make_site(int(n[i]), int(dims[i]), int(r.integers(12, 41)), case["chunks"], seed * 1000 + i)
                           for i in range(case["sites"]))


def _window(case, seed):
    """Sites and features of a time-drift window: spikes near a site have their second site beside it."""
    r = np.random.default_rng(seed)
    n, d, S = case["n"], case["d"], case["sites"]
    s1 = r.integers(1, S + 1, n)
    s2 = np.clip(s1 + r.choice([-1, 1], n), 1, S)
    units = r.normal(0.0, 10.0, (3 * S, d))
    lab = 3 * (s1 - 1) + r.integers(0, 3, n)
    f1 = units[lab] + r.normal(0.0, 1.2, (n, d))
    f2 = 0.6 * f1 + r.normal(0.0, 1.2, (n, d))
    return np.concatenate([s1, s2]).astype(np.int32), f1.astype(np.float32), f2.astype(np.float32)


def _chunk(case, seed):
    """The middle chunk of a site whose chunks are all linked: (F, rho, runs, vnConst)."""
    F, plan = _site(case, seed)
    i = len(plan["q0"]) // 2
    r0, r1 = int(plan["roff"][i]), int(plan["roff"][i + 1])
    vn = [case["d"], F.shape[0], r1 - r0, int(plan["q0"][i]), int(plan["nq"][i])]
    rho = np.random.default_rng(seed + 5).uniform(0.05, 0.5, F.shape[0]).astype(np.float32)
    return F, rho, np.ascontiguousarray(plan["rs"][r0:r1]), np.ascontiguousarray(plan["rn"][r0:r1]), vn


def _v4(case, seed):
    F = synth.make_site(case["n"], case["d"], case["clusters"], 1, seed)["F"]
    r = np.random.default_rng(seed + 9)
    a = int(r.integers(0, case["n"] - case["n_own"] + 1))
    return F, r.uniform(0.05, 0.5, case["n"]).astype(np.float32), np.arange(case["n"]), np.arange(a, a + case["n_own"])


def _linkage(case, seed):
    """Amplitudes and positions of a recording whose units drift slowly along the probe."""
    r = np.random.default_rng(seed)
    n, S = case["n"], case["sites"]
    unit = r.integers(0, 4 * S, n)
    t = np.linspace(0.0, 6.0, n)
    pos = 20.0 * S * r.random(4 * S)[unit] + 15.0 * np.sin(t) + r.normal(0.0, 4.0, n)
    amp = 30.0 + 200.0 * r.random(4 * S)[unit] + r.normal(0.0, 10.0, n)
    return amp.astype(np.float32), pos.astype(np.float32)


def _stream(case, seed):
    """The recording's layout goes with the case, its spikes with the seed."""
    wl = stream.make_workload(case["sites"], case["n"], case["chunks"], case["d"])
    r = np.random.default_rng(seed)
    F = wl["F16"].numpy()
    F[:] = F[:, r.permutation(case["d"])] + 0.25 * r.standard_normal(F.shape, np.float32)
    return wl


def prepare(case, seed):
    kind = case["kind"]
    dev = lambda *a: [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in a]
    st = dict(case=case)
    if kind in ("site", "clusters"):
        F, plan = _site(case, seed)
        st["F"], = dev(F)
        st["plan"] = irc.Plan(plan)
        if case.get("copies", 0):
            st["rho_copies"], = dev(_rho_copies(case, seed))
    elif kind == "probe":
        b = _probe(case, seed)
        st["F"], = dev(b.F)
        st["plan"] = b.make_plan()
    elif kind == "chunk":
        F, rho, rs, rn, vn = _chunk(case, seed)
        st["F"], st["rho"], st["rs"], st["rn"] = dev(F, rho, rs, rn)
        st["vn"] = vn
    elif kind == "v4":
        F, rho, vi2, vi1 = _v4(case, seed)
        st["F"], st["rho"], st["vi2"], st["vi1"] = dev(F, rho, vi2, vi1)
    elif kind == "window":
        st["site"], st["f1"], st["f2"] = dev(*_window(case, seed))
        st["dc2"] = _dc2(case)
    elif kind == "linkage":
        st["amp"], st["pos"] = dev(*_linkage(case, seed))
    else:
        st["streamer"] = stream.Streamer(_stream(case, seed), KNN, case["mode"])
    return st


def _rho_copies(case, seed):
    return np.random.default_rng(seed + 3).uniform(0.05, 0.5, case["copies"]).astype(np.float32)


def _dc2(case):
    return float(np.float32(2.2 * case["d"]))


# ---- one pass ----------------------------------------------------------------------------------------------------------------------

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("site", "probe", "clusters"):
        if case.get("copies", 0):
            o = irc.site_knn(st["plan"], st["F"], KNN, case["mode"])
            R = torch.cat([o["rho"], st["rho_copies"]])
            o["delta"], o["nneigh"] = irc.site_delta(st["plan"], st["F"], R, case["mode"], 512, KNN, o["miKnn"], o["d2Knn"])
        else:
            o = irc.knn_rho_delta_site(st["plan"], st["F"], KNN, case["mode"])
        out = [o[k] for k in ("vrKnn", "rho", "miKnn", "d2Knn", "delta", "nneigh") if o[k] is not None]
        if kind == "clusters":
            rho, order = irc.sort_rho(o["rho"])
            c = irc.assign_cluster_knn(rho, o["delta"], order, o["nneigh"], o["miKnn"], 1.0, 30)
            pad = lambda x: torch.nn.functional.pad(x, (0, case["n"] - c["nClu"]))    # as many values whatever the cluster count
            out += [rho, order, c["viClu"], pad(c["icl"]), pad(c["vnSpk_clu"])]
        return out
    if kind == "chunk":
        D, I = irc.search_min_drift(st["F"], st["rs"], st["rn"], st["vn"], 1024)
        E, J = irc.search_delta_drift(st["F"], st["rho"], st["rs"], st["rn"], st["vn"], 512)
        return [D, I, E, J]
    if kind == "v4":
        K, I = irc.cuda_knn(st["F"], st["vi2"], st["vi1"], KNN)
        D, N = irc.cuda_delta_knn_host(st["F"], st["rho"], st["vi2"], st["vi1"])
        return [K, I, D, N]
    if kind == "window":
        n = case["n_own"]
        rho = irc.rho_drift(st["site"], st["f1"], st["f2"], n, st["dc2"])
        rho12 = rho.repeat(-(-case["n"] // n))[:case["n"]]           # the other chunks' rho is at hand in a real pass
        D, N = irc.delta_drift(st["site"], st["f1"], st["f2"], rho12, n, st["dc2"])
        return [rho, D, N]
    if kind == "linkage":
        return list(irc.calc_drift(st["amp"], st["pos"], case["sites"], case["chunks"], case["batch"]))
    s = st["streamer"]
    s.run()
    return [s.out[k] for k in ("rho", "delta", "nneigh", "miKnn")]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------

def _site_pairs(case):
    n, c = case["n"], case["chunks"]
    return n * (n + case.get("copies", 0)) * min(LINKS, c) / c


def work(case):
    kind, n, d = case["kind"], case["n"], case.get("d", 25)
    if kind in ("site", "clusters"):
        m = n + case.get("copies", 0)
        out = n * (16 + 4 * KNN * (1 if case["mode"] == "ref" else 2)) + (n * 16 if kind == "clusters" else 0)
        return dict(bytes=4 * d * m + out, flops=2 * d * _site_pairs(case))
    if kind == "probe":                                              # spikes spread over the sites as exp(N(0, 1)): E[x^2] / E[x]^2 = e
        return dict(bytes=n * (4 * d + 16 + 8 * KNN), flops=2 * d * math.e * n * n / case["sites"] * min(LINKS, case["chunks"]) / case["chunks"])
    if kind == "chunk":
        nq = n / case["chunks"]
        return dict(bytes=4 * d * n + 4 * n + nq * (1024 + 512) * 8, flops=2 * 2 * d * nq * n)
    if kind == "v4":
        return dict(bytes=4 * (d + 1) * n + case["n_own"] * (KNN + 3) * 8, flops=2 * 2 * d * n * case["n_own"])
    if kind == "window":
        return dict(bytes=n * (8 * d + 12), flops=2 * 2 * d * case["n_own"] * n * 2 / case["sites"])
    if kind == "linkage":
        return dict(bytes=8 * n, flops=3 * case["chunks"] * min(case["chunks"], 256) * 10 * case["sites"])
    return dict(bytes=n * (2 * d + 12 + 4 * KNN), flops=2 * d * math.e * n * n / case["sites"] * LINKS / case["chunks"])


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------------

def _d2(A, B):
    """Squared distances in FP64; copies of the query (and the query) at infinity."""
    d = (A * A).sum(1)[:, None] + (B * B).sum(1)[None] - 2.0 * (A @ B.T)
    return d


def _runs64(plan, i, dev):
    r0, r1 = int(plan["roff"][i]), int(plan["roff"][i + 1])
    rs, rn = torch.as_tensor(plan["rs"][r0:r1]).long().to(dev), torch.as_tensor(plan["rn"][r0:r1]).long().to(dev)
    off = torch.arange(int(plan["rn"][r0:r1].sum()), device=dev) - torch.repeat_interleave(torch.cumsum(rn, 0) - rn, rn)
    run = torch.repeat_interleave(torch.arange(r1 - r0, device=dev), rn)
    return rs[run] + off, run, off, r1 - r0


def _bin_min(d, run, off, n_runs, nT):
    """Minima of the reference's nT bins of every row: bin t scans run t % n_runs from t // n_runs in steps of nT // n_runs."""
    step = nT // n_runs
    out = torch.full((d.shape[0], nT), SINGLE_INF, dtype=torch.float64, device=d.device)
    t = (off % step) * n_runs + run
    out.scatter_reduce_(1, t.expand(d.shape[0], -1), d, "amin")
    t2 = step * n_runs + run
    m = (off >= step) & (off % step == 0) & (t2 < nT)
    if bool(m.any()):
        out.scatter_reduce_(1, t2[m].expand(d.shape[0], -1), d[:, m], "amin")
    return out


def _knn64(F, plan, mode, R_more):
    """vrKnn, rho, d2Knn, delta of every query in FP64 (the reference's bins for mode "ref")."""
    dev = "cuda"
    X = torch.from_numpy(F).to(dev).double()
    n, qb = plan["n_out"], plan["q_base"]
    d2k = torch.full((n, KNN), SINGLE_INF, dtype=torch.float64, device=dev)
    cuts = [(int(q0) + a, min(4096, int(nq) - a), i) for i, (q0, nq) in enumerate(zip(plan["q0"], plan["nq"])) for a in range(0, int(nq), 4096)]

    def dist(q, m, i):
        c, run, off, nr = _runs64(plan, i, dev)
        d = _d2(X[q:q + m], X[c])
        return torch.where(d > 1e-8, d, torch.full_like(d, SINGLE_INF)), c, run, off, nr

    for q, m, i in cuts:
        d, c, run, off, nr = dist(q, m, i)
        if mode == "ref":
            d = _bin_min(d, run, off, nr, 1024)
        k = min(KNN, d.shape[1])
        d2k[q - qb:q - qb + m, :k] = torch.topk(d, k, dim=1, largest=False, sorted=True).values
    vr = d2k[:, -1].sqrt()
    rho = 1.0 / vr
    R = rho if R_more is None else torch.cat([rho, torch.from_numpy(R_more).to(dev).double()])
    delta = torch.empty_like(rho)
    for q, m, i in cuts:
        d, c = dist(q, m, i)[:2]
        d = torch.where(R[c][None] > R[q:q + m, None], d, torch.full_like(d, SINGLE_INF))
        delta[q - qb:q - qb + m] = d.amin(1).sqrt() * R[q:q + m]
    return vr, rho, d2k, delta


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linkage", "stream"):
        return None                                                  # whole numbers alone; rows of a ring that the pass itself lays out
    if kind in ("site", "probe", "clusters"):
        if kind == "probe":
            b = _probe(case, seed)
            F, plan, more = b.F, b.plan, None
        else:
            F, plan = _site(case, seed)
            more = _rho_copies(case, seed) if case.get("copies", 0) else None
        vr, rho, d2k, delta = _knn64(F, plan, case["mode"], more)
        out = [vr, rho, None] + ([d2k] if case["mode"] != "ref" else []) + [delta, None]
        return out + ([rho / rho.max(), None, None, None, None] if kind == "clusters" else [])
    if kind == "chunk":
        F, rho, rs, rn, vn = _chunk(case, seed)
        plan = dict(rs=rs, rn=rn, roff=np.array([0, len(rs)]))
        X, R = torch.from_numpy(F).cuda().double(), torch.from_numpy(rho).cuda()
        c, run, off, nr = _runs64(plan, 0, "cuda")
        q = slice(vn[3], vn[3] + vn[4])
        d = _d2(X[q], X[c])
        d = torch.where(d > 1e-8, d, torch.full_like(d, SINGLE_INF))
        e = torch.where(R[c][None] > R[q, None], d, torch.full_like(d, SINGLE_INF))
        return [_bin_min(d, run, off, nr, 1024).sqrt(), None, _bin_min(e, run, off, nr, 512).sqrt(), None]
    if kind == "v4":
        F, rho, vi2, vi1 = _v4(case, seed)
        X, R = torch.from_numpy(F).cuda().double(), torch.from_numpy(rho).cuda()
        d = _d2(X[vi1], X[vi2]).clamp_(min=0.0)
        j = torch.arange(case["n"], device="cuda")
        K = _bin_min(d, torch.zeros_like(j), j, 1, 512).sort(1).values[:, KNN - 1].sqrt()
        e = torch.where(R[vi2][None] > R[vi1, None], d, torch.full_like(d, SINGLE_INF))
        return [K, None, e.amin(1).sqrt(), None]
    site, f1, f2 = _window(case, seed)
    n, n1, dc2 = case["n"], case["n_own"], _dc2(case)
    site = torch.from_numpy(site).cuda()
    A, B = torch.from_numpy(f1).cuda().double(), torch.from_numpy(f2).cuda().double()
    s1, s2, sq = site[:n][None], site[n:][None], site[:n1, None]
    d = torch.where(s1 == sq, _d2(A[:n1], A), _d2(A[:n1], B)).clamp_(min=0.0)
    hit = (s1 == sq) | (s2 == sq)
    rho = ((d <= dc2) & hit).sum(1).double() / hit.sum(1).double()
    r12 = rho.float().repeat(-(-n // n1))[:n]
    d = torch.where(hit & (r12[None] > r12[:n1, None]), d, torch.full_like(d, SINGLE_INF))
    return [rho, (d.amin(1) / dc2).sqrt(), None]
