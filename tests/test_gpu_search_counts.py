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
