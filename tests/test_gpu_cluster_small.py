"""Label propagation of a small site in one block against the oracle, at the
sizes where its form changes, with chains as long as the site and passes up to
the cap."""
import numpy as np
import pytest

from ironclust_gb300 import irc
from oracle import oracle as O
from tests.cluster_cases import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chain", ["random", "chain", "backward"])
@pytest.mark.parametrize("n", [40, 1023, 1025, 4095, 4096, 4097])
def test_propagation_matches_oracle(gpu, n, chain):
    rho, delta, ordrho, nneigh, mk = random_case(n, n=n, p_quirk=0.3, delta_scale=1.1)
    nneigh = nneigh.copy()
    if chain == "chain":                                       # every spike's neighbour is the one ranked before it
        nneigh[ordrho[1:] - 1] = ordrho[:-1]
    if chain == "backward":                                    # ... behind it: a rank more per pass
        nneigh[ordrho[:-1] - 1] = ordrho[1:]
    for min_count in (0, 5):
        ref = O.assign_cluster_knn(rho, delta, ordrho, nneigh, mk, 1.0, min_count)
        out = irc.assign_cluster_knn(rho, delta, ordrho, nneigh, mk, 1.0, min_count)
        for k in ("nClu", "nClu_pre", "nClu_post"):
            assert out[k] == ref[k], k
        for k in ("viClu", "icl", "vnSpk_clu"):
            np.testing.assert_array_equal(out[k].cpu().numpy(), ref[k], err_msg=k)
