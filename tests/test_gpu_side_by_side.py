"""Small ensembles advanced side by side run two chains per warp, alone one; the state
and the sums do not depend on it."""
import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu
KAP = (0.0, 2.0e-3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("kw", [dict(nk=50), dict(nk=50, kappa=KAP),
                                dict(nk=50, eq_type=1, corr_p=16, corr_m=2, sync_dt=1.0, t_end=100.0)], ids=str)
def test_side_by_side(dsm_mod, kw):
    a = [dsm_mod.Ensemble(n_chains=1500, seed=191, stream=i, **kw) for i in range(3)]
    b = [dsm_mod.Ensemble(n_chains=1500, seed=191, stream=i, lanes_per_chain=32, **kw) for i in range(3)]
    for x in a + b:
        x.init_equilibrium()
    assert a[0].step_kernel()["lanes"] == 32
    t = 0.0
    for _ in range(3):
        t += 20.0
        for x in a:
            x.advance_start(t)
        ev = [None] * 3
        while any(e is None for e in ev):
            ev = [x.poll() if e is None else e for x, e in zip(a, ev)]
        assert [e[0] for e in ev] == [y.advance(t) for y in b]
    assert [x.step_kernel()["lanes"] for x in a] == [16] * 3
    for _ in range(2):  # the launch after one that ran alone
        t += 2.0
        for x, y in zip(a, b):
            assert x.advance(t) == y.advance(t)
    assert [x.step_kernel()["lanes"] for x in a] == [32] * 3
    for x, y in zip(a, b):
        x.advance_series(1.0, 2)
        y.advance_series(1.0, 2)
        assert_bitexact(gpu_state(x), gpu_state(y), what="side by side")
        if "eq_type" in kw:
            assert np.array_equal(x.gt_raw()[0], y.gt_raw()[0])


def test_destroyed_while_under_way(dsm_mod):
    """A handle that goes away with a launch pending no longer counts."""
    a, b = (dsm_mod.Ensemble(nk=50, n_chains=1500, seed=192) for _ in range(2))
    for x in (a, b):
        x.init_equilibrium()
    b.advance_start(5.0)
    b.close()
    for t in (1.0, 2.0):
        a.advance(t)
    assert a.step_kernel()["lanes"] == 32
