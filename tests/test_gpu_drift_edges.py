"""The device drift linkage where its selection and histograms change form,
against the numpy restatement: one value only, more edges than the blocks count
in shared memory, a subsample that drops positions, fewer spikes than a block,
chunks of several parts, more bins than shared memory holds, values that are not
finite."""
import numpy as np
import pytest

from ironclust_gb300 import irc
from oracle import drift_oracle as DO

pytestmark = pytest.mark.gpu

# spikes, sites, chunks, linked chunks, amplitude quantiles, values
CASES = [
    (300, 4, 20, 5, 10, "plain"), (5000, 16, 40, 15, 10, "one value"), (60000, 64, 300, 15, 10, "few values"),
    (100001, 128, 60, 15, 10, "plain"), (254321, 32, 40, 7, 10, "plain"), (199999, 1, 50, 10, 1, "plain"),
    (150000, 200, 60, 10, 50, "plain"), (400000, 16, 20, 5, 10, "few values"), (30000, 1024, 30, 5, 3, "plain"),
    (30000, 24, 30, 6, 1024, "plain"), (50000, 24, 40, 8, 10, "not finite"),
]


@pytest.mark.parametrize("n,sites,chunks,batch,quantiles,values", CASES)
def test_calc_drift_edges(gpu, n, sites, chunks, batch, quantiles, values):
    rng = np.random.default_rng(n)
    amp = rng.gamma(3.0, 40.0, n).astype(np.float32)
    pos = (20.0 * rng.integers(0, 8 * max(sites // 8, 1), n) + rng.normal(0, 6.0, n)).astype(np.float32)
    if values == "one value":
        amp[:], pos[:] = 7.5, -3.0
    if values == "few values":
        amp, pos = np.round(amp / 50.0).astype(np.float32), np.round(pos / 100.0).astype(np.float32)
    if values == "not finite":
        amp[::17], pos[5::23], pos[3::101] = np.inf, -np.inf, np.float32(-0.0)
    kw = dict(nTime_drift=chunks, nTime_batch=batch, nQuantile_drift=quantiles)
    lim_o, ml_o = DO.calc_drift(amp, pos, sites, **kw)
    lim_d, ml_d = irc.calc_drift(amp, pos, sites, **kw)
    assert np.array_equal(lim_d, lim_o)
    assert np.array_equal(ml_d, ml_o)
