"""Ensemble sums and the pooled |Q| list at sizes around the reductions' strides
(256 partial sums, 8 rows in flight, 1024 runs of chains)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAP = (0.0, 2.0e-3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1023, 1025, 2049, 5000, 39000])
def test_sums_and_lists(dsm_mod, n):
    e = dsm_mod.Ensemble(nk=30, n_chains=n, seed=95)
    e.init_equilibrium()
    e.advance(3.0)
    heads, qn, _ = e.get_chains()
    Z = heads["Z"].astype(int)
    m = (np.arange(qn.shape[1])[None, :] >= 1) & (np.arange(qn.shape[1])[None, :] < Z[:, None] - 1)
    q = qn[m].astype(np.float32)
    hz, hn, got = e.distributions()
    assert len(got) == np.maximum(Z - 2, 0).sum()
    # |Q| by three roundings of squares and sums and one of the root
    want = np.sort(np.sqrt((q[:, :3].astype(np.float64) ** 2).sum(axis=1)))
    assert np.allclose(got, want, rtol=4 * 2.0**-24, atol=0.0)
    assert hz.sum() == n
    s, cnt = e.stress()
    assert cnt == n and np.float32(s[7]) == np.float32(Z.sum() / n)


@pytest.mark.parametrize("n", [1, 257, 2049, 4100])
def test_series_equals_single_windows(dsm_mod, n):
    kw = dict(nk=30, n_chains=n, kappa=KAP, seed=96)
    a, b = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(**kw)
    for x in (a, b):
        x.init_equilibrium()
    _, rows = a.advance_series(0.75, 5)
    for k in range(5):
        b.advance(0.75 * (k + 1))
        s, cnt = b.stress()
        assert cnt == n and np.array_equal(np.float32(rows[k]), np.float32(s))
