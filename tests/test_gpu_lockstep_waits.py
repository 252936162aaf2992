"""A wait between the warps of a lockstep launch that runs out: the advance fails, the
clock stays, calls that need the chains are refused, and new chains run as if
nothing had been.  With the default limit a warp whose chains all wait goes on."""
import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu
N = 7400


def test_wait_that_runs_out(dsm_mod, oracle_mod, tmp_path):
    kw = dict(nk=200, n_chains=N, seed=181)
    g = dsm_mod.Ensemble(eq_type=1, sync_dt=0.5, t_end=100.0, corr_p=16, corr_m=2, **kw)
    g.init_equilibrium()
    g.advance(0.5)
    g.set_wait_polls(1)  # no request is served within two polls of the launch's start
    with pytest.raises(dsm_mod.DSMError, match="ran out"):
        g.advance(30.0)
    g.set_wait_polls(0)
    refused = [lambda: g.advance(4.0), lambda: g.advance_start(4.0), lambda: g.advance_series(1.0, 2),
               lambda: g.autotune(1.0), g.get_chains, g.get_ext, g.stress, g.gt, g.gt_raw, g.distributions, g.r1,
               lambda: g.save(str(tmp_path / "c")), lambda: g.checkpoint(str(tmp_path / "k")),
               lambda: dsm_mod.advance_batch([g], 4.0)]
    for call in refused:
        with pytest.raises(dsm_mod.DSMError, match="set them anew"):
            call()
    o = oracle_mod.Oracle(corr=True, sync_dt=0.5, t_end=100.0, corr_p=16, corr_m=2, **kw)
    g.init_equilibrium()
    o.init_equilibrium()
    assert g.advance(30.0) == o.run(30.0)
    assert g.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(g), o.get_state(), what="after a lost launch")


def test_batch_keeps_the_other_groups(dsm_mod):
    """Only the group whose launch gave up is lost."""
    kw = dict(nk=40, n_chains=600, seed=182)
    a = dsm_mod.Ensemble(nk=200, n_chains=N, seed=182)
    b, c = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(**kw)
    for x in (a, b, c):
        x.init_equilibrium()
    a.set_wait_polls(1)
    with pytest.raises(dsm_mod.DSMError):
        dsm_mod.advance_batch([b, a], 20.0)
    with pytest.raises(dsm_mod.DSMError, match="set them anew"):
        a.get_chains()
    c.advance(20.0)
    assert_bitexact(gpu_state(b), gpu_state(c), what="other group")
    assert b.advance(21.0) == c.advance(21.0)


def test_short_limit_with_progress(dsm_mod):
    """Chains that wait for their earlier time slices longer than the limit: the launch
    makes progress meanwhile, so no wait gives up (a limit of some ten milliseconds,
    a launch of several hundred)."""
    kw = dict(nk=300, beta=0.5, n_chains=6000, seed=183)
    a, b = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    a.set_wait_polls(1 << 17)
    assert a.advance(600.0) == b.advance(600.0)
    assert_bitexact(gpu_state(a), gpu_state(b), what="short limit")
    heads, _, _ = a.get_chains()
    assert np.all(heads["stall_flag"] == 0)
