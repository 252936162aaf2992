"""Default lanes per chain of ensembles with per-chain N_K: two chains per warp when
there is work enough and the middle class is small or fills its slots, else one;
the state does not depend on it."""
import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,low,high,many,eq_type,lanes", [
    (9000, 20, 40, 0, 1, 16),       # one slot size, no classes
    (9000, 150, 300, 40, 1, 16),    # a middle class of 40 chains
    (9000, 150, 300, 40, 0, 16),
    (9000, 150, 300, 900, 1, 32),   # a middle class that holds the other up
    (4000, 20, 40, 0, 1, 32),       # too little work
    (9000, 150, 300, 40, 9, 32),    # flow
], ids=str)
def test_poly_default_lanes(dsm_mod, n, low, high, many, eq_type, lanes):
    nkc = np.full(n, low, np.int32)
    nkc[:: n // many if many else n] = high
    kw = dict(nk=int(nkc.max()), nk_chain=nkc, n_chains=n, seed=81, sync_dt=0.5, t_end=100.0, corr_p=16, corr_m=2)
    if eq_type == 9:
        kw["kappa"] = (0.0, 2.0e-3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)
    else:
        kw["eq_type"] = eq_type
    a = dsm_mod.Ensemble(**kw)
    b = dsm_mod.Ensemble(lanes_per_chain=48 - lanes, **kw)
    for x in (a, b):
        x.init_equilibrium()
    sched = [k for k in a.schedule() if k["chains"] > 0]
    if sched:
        assert sched[-1]["lanes"] == lanes
    for t in (1.0, 2.5):
        assert a.advance(t) == b.advance(t)
    assert_bitexact(gpu_state(a), gpu_state(b), what=f"{lanes} lanes")
    if eq_type == 1:
        assert np.array_equal(a.gt_raw()[0], b.gt_raw()[0])
