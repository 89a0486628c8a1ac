"""Work items split over their candidates (irc_tc.cu) against the same search
with whole ones, bit for bit: 128-candidate units are never split, nor items of
a plan on a buffer without room for it."""
import ctypes as C

import numpy as np
import pytest
import torch

from ironclust_gb300 import _lib, irc
from tests.cases import small_site

pytestmark = pytest.mark.gpu

# queries, features, chunk sizes or their number, copies: few items of a window just wide enough and of a wide one,
# more than a turn of the machine with a few left over, items with windows of different widths, a window beyond
# 512 tiles, exact copies that overflow lists
SHAPES = [
    (3072, 18, 1, False), (3300, 24, 1, False), (5000, 33, 7, True), (9999, 45, 1, False), (20000, 24, 1, False),
    (45000, 12, 20, False), (30011, 33, 12, True), (66000, 6, 1, False), (8000, 54, 2, False), (6500, 24, 1, False),
]


@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("n,d,chunks,secondary", SHAPES)
def test_split_items_equal_whole_ones(gpu, n, d, chunks, secondary, dup):
    F, plan, _ = small_site(n=n, d=d, n_chunks=chunks, seed=n % 97, n_dup=n // 8 if dup else 0, secondary=secondary)
    if dup:
        F[: n // 20] = F[0]                                    # more copies than a list holds
    Fd = torch.from_numpy(np.ascontiguousarray(F)).to(gpu)
    P, Q, W = irc.Plan(plan), irc.Plan(plan), irc.Plan(plan)
    _lib.check(_lib.lib().irc_plan_tc_units(Q.h, 128), "irc_plan_tc_units")
    # (a buffer of the caller's that has no room for the parts: the same items whole)
    size = _lib.lib().irc_plan_tc_bytes(P.h, d)
    buf = torch.empty(size, dtype=torch.uint8, device=gpu)
    _lib.check(_lib.lib().irc_plan_set_tc_buffer(W.h, C.c_void_p(buf.data_ptr()), C.c_size_t(size - 256)), "irc_plan_set_tc_buffer")
    try:
        irc.site_knn(W, Fd, 30, "bf16")
    except _lib.IrcError:                                      # (not a plan with split items)
        W = P
    for mode, whole in (("exact", Q), ("ref", Q), ("bf16", W)):
        for _ in range(2):                                     # (the second call on used memory)
            a = irc.site_knn(P, Fd, 30, mode)
        b = irc.site_knn(whole, Fd, 30, mode)
        for k in ("miKnn", "vrKnn", "d2Knn"):
            if a[k] is not None:
                assert torch.equal(a[k].view(torch.int32), b[k].view(torch.int32)), (mode, k)
