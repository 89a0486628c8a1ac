"""Plans whose chunks do not ascend: queries that ordered scans finish (more
equal distances than a list holds) are searched in their own chunk's window."""
import numpy as np
import pytest
import torch

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cases import small_site

pytestmark = pytest.mark.gpu


def reorder(plan, order):
    runs = [np.arange(plan["roff"][i], plan["roff"][i + 1]) for i in order]
    i32 = lambda a: np.asarray(a, np.int32)
    return dict(plan, q0=i32(plan["q0"][order]), nq=i32(plan["nq"][order]), roff=i32(np.concatenate([[0], np.cumsum([len(r) for r in runs])])),
                rs=i32(np.concatenate([plan["rs"][r] for r in runs])), rn=i32(np.concatenate([plan["rn"][r] for r in runs])))


@pytest.mark.parametrize("n,chunks", [(2400, 6), (9000, 9)])
@pytest.mark.parametrize("mode", ["exact", "bf16"])
def test_chunks_in_any_order(gpu, n, chunks, mode):
    F, plan, _ = small_site(n=n, d=6, seed=n, sizes=[n // chunks] * chunks, n_dup=0)
    F = np.round(F / 8.0).astype(np.float32)                   # hundreds of equal distances
    want, d2 = O.exact_knn_f32(F, plan, 30)
    Fd = torch.from_numpy(F).to(gpu)
    for order in (np.arange(chunks), np.arange(chunks)[::-1], np.random.default_rng(1).permutation(chunks)):
        P = irc.Plan(reorder(plan, order))
        got = irc.site_knn(P, Fd, 30, mode)
        assert P.search_counts()["scans"] > 0 or n < 9000      # (windows of 1,200 rows may hold them)
        if mode == "exact":
            assert np.array_equal(got["miKnn"].cpu().numpy(), want)
        assert np.array_equal(got["d2Knn"].cpu().numpy().view(np.int32), d2.view(np.int32))
