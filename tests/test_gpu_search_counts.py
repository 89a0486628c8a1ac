"""Where a plan's calls went (irc_plan_search_counts)."""
import ctypes as C

import numpy as np
import pytest
import torch

from ironclust_gb300 import _lib, irc
from tests.cases import small_site

pytestmark = pytest.mark.gpu


def flush(gpu):
    torch.empty(256 << 20, dtype=torch.uint8, device=gpu).zero_()


# a few items left of a full turn, half a machine of them, windows beyond 512 tiles
@pytest.mark.parametrize("n,d,chunks", [(20000, 24, 1), (45000, 12, 20), (66000, 6, 1)])
def test_split_items_leave_what_whole_ones_leave(gpu, n, d, chunks):
    """The second pass of a split item reads the thresholds it was given, also
    when its query tile lands late (cold caches): a lost threshold empties the
    item's lists, and its queries would be finished by ordered scans."""
    F, plan, _ = small_site(n=n, d=d, n_chunks=chunks, seed=5, n_dup=0)
    Fd = torch.from_numpy(np.ascontiguousarray(F)).to(gpu)
    P, W = irc.Plan(plan), irc.Plan(plan)
    # (a buffer of the caller's that has no room for the parts: the same items whole)
    size = _lib.lib().irc_plan_tc_bytes(P.h, d)
    buf = torch.empty(size, dtype=torch.uint8, device=gpu)
    _lib.check(_lib.lib().irc_plan_set_tc_buffer(W.h, C.c_void_p(buf.data_ptr()), C.c_size_t(size - 256)), "irc_plan_set_tc_buffer")
    irc.site_knn(W, Fd, 30, "bf16")
    whole = W.search_counts()["scans"]
    for _ in range(10):
        flush(gpu)
        irc.site_knn(P, Fd, 30, "bf16")
        assert P.search_counts()["scans"] == whole


def ragged(n_long, short, n_short):
    """One chunk of n_long spikes, then n_short chunks of `short`; every window is the chunk itself."""
    sizes = np.array([n_long] + [short] * n_short, np.int32)
    q0 = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    n = int(sizes.sum())
    return dict(q0=q0, nq=sizes, roff=np.arange(len(sizes) + 1, dtype=np.int32), rs=q0, rn=sizes, q_base=0, n_out=n, n_f=n)


def test_split_rule_looks_at_the_items_it_splits(gpu):
    """Items behind the last full turn are split when they are long, not when
    another chunk's are: one wide window (157 items) before 200 of one tile."""
    plan = ragged(20000, 100, 200)
    F = torch.from_numpy(small_site(n=plan["n_f"], d=24, n_chunks=1, seed=9)[0]).to(gpu)
    P = irc.Plan(plan)
    irc.site_knn(P, F, 30, "bf16")
    assert P.search_counts()["splits"] == 0
    # chunk order, the short chunks first: the rest are items of the wide window
    back = dict(plan, **{k: np.concatenate([plan[k][1:], plan[k][:1]]) for k in ("q0", "nq", "rs", "rn")})
    Q = irc.Plan(back)
    _lib.check(_lib.lib().irc_plan_tc_layout(Q.h, 1, 1), "irc_plan_tc_layout")
    irc.site_knn(Q, F, 30, "bf16")
    assert Q.search_counts()["splits"] == 357 - 2 * 152
    R = irc.Plan(ragged(20000, 100, 0))
    irc.site_knn(R, F[:20000], 30, "bf16")
    assert R.search_counts()["splits"] == 157 - 152
