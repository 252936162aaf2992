"""The lockstep step kernel (large monodisperse equilibrium ensembles) against the
oracle and against the 16-lane tiles, bit for bit: every built slot size (pairs
per sub-chunk of the pick and lanes per chain), capacity refusals, CD off, the GEX
background, both correlator kinds across several sample buffers, chains that
outgrow their slot, and an abort."""
import threading

import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu
N = 7400  # more than 48 chains per SM: the lockstep kernel runs


@pytest.mark.parametrize("kw", [
    dict(nk=100, beta=10.0),            # 2 pairs per sub-chunk
    dict(nk=90, beta=3.0),              # 3
    dict(nk=100),                       # 5, build for 6 blocks per SM
    dict(nk=131),                       # 9
    dict(nk=170, beta=0.5),             # 8 lanes per chain, 8 pairs
    dict(nk=463, beta=0.5),             # 8 lanes per chain, 12 pairs
    dict(nk=100, cd_flag=0),
    dict(nk=100, z_max=52),             # creations refused at capacity
    dict(nk=100, gex=(1.0, 1.0, 1000.0, 100.0)),
], ids=str)
def test_lockstep_bitexact(dsm_mod, oracle_mod, kw):
    gex = kw.get("gex")
    okw = {k: v for k, v in kw.items() if k != "gex"}
    if gex is not None:
        okw["gex_tables"] = dsm_mod.gex_tables(*gex, 1.0)
    g = dsm_mod.Ensemble(n_chains=N, seed=71, **kw)
    o = oracle_mod.Oracle(n_chains=N, seed=71, **okw)
    g.init_equilibrium()
    o.init_equilibrium()
    for t in (0.5, 2.0):
        assert g.advance(t) == o.run(t)
    assert_bitexact(gpu_state(g), o.get_state(), what=f"lockstep {kw}")
    ev = g.advance(1.0e9, step_limit=400)
    assert ev == o.run(1.0e9, step_limit=400)
    assert_bitexact(gpu_state(g), o.get_state(), what=f"lockstep {kw}, event limit")


@pytest.mark.parametrize("kw", [dict(nk=151, eq_type=1, corr_p=16, corr_m=2),
                                dict(nk=200, eq_type=1, corr_p=64, corr_m=8),
                                dict(nk=204, beta=0.5, eq_type=1, corr_p=96, corr_m=4),
                                dict(nk=150, eq_type=2, corr_p=64, corr_m=8),
                                dict(nk=151, eq_type=2, corr_p=8, corr_m=2)], ids=str)
def test_lockstep_correlator_equals_tiles(dsm_mod, kw):
    """States, G(t) or MSD sums and R1 over windows that end inside, at and after
    full sample buffers (80 and 7 samples per window)."""
    a = dsm_mod.Ensemble(n_chains=N, seed=72, sync_dt=0.25, t_end=4000.0, **kw)
    b = dsm_mod.Ensemble(n_chains=N, seed=72, sync_dt=0.25, t_end=4000.0, lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    for t in (20.0, 21.75, 53.75):
        assert a.advance(t) == b.advance(t)
        ga, ca = a.gt_raw()
        gb, cb = b.gt_raw()
        assert np.array_equal(ca, cb) and np.array_equal(ga, gb)
    assert_bitexact(gpu_state(a), gpu_state(b), what=f"lockstep {kw}")
    assert np.array_equal(a.r1(), b.r1())


@pytest.mark.parametrize("eq_type", [0, 1])
def test_lockstep_overflow_and_abort(dsm_mod, oracle_mod, eq_type):
    """Slots a little above the mean strand count: many chains finish in the
    overflow launch; then a launch that is told to abort before it starts."""
    kw = dict(nk=151, n_chains=N, seed=73)
    g = dsm_mod.Ensemble(eq_type=eq_type, sync_dt=1.0, t_end=100.0, corr_p=16, corr_m=2, **kw)
    o = oracle_mod.Oracle(**kw)
    g.set_schedule(small_slot=80, z_margin_sd=0.01)
    g.init_equilibrium()
    o.init_equilibrium()
    deferred = 0
    for t in (1.0, 3.0):
        g.advance(t)
        o.run(t)
        deferred += g.window_stats()["deferred"]
    assert deferred > N // 20
    assert_bitexact(gpu_state(g), o.get_state(), what="lockstep overflow")
    assert g.advance(50.0, abort=np.ones(1, np.int32)) == -1
    assert_bitexact(gpu_state(g), o.get_state(), what="lockstep abort")


@pytest.mark.parametrize("kw", [dict(nk=300, beta=0.5, eq_type=0),
                                dict(nk=300, beta=0.5, eq_type=1, corr_p=64, corr_m=8),
                                dict(nk=230, beta=0.4, eq_type=2, corr_p=16, corr_m=2),
                                dict(nk=300, beta=0.5, eq_type=1, corr_p=64, corr_m=8, small_slot=206)], ids=str)
def test_lockstep_time_slices(dsm_mod, kw):
    """Launches in time slices (8 lanes per chain, more chains than slots, windows of
    thousands of events) against the tiles: windows with and without slices, between
    samples and with part-filled sample buffers, a series of windows, and chains that
    outgrow their slot."""
    kw = dict(kw)
    small = kw.pop("small_slot", 0)
    n = 6000
    a = dsm_mod.Ensemble(n_chains=n, seed=74, sync_dt=0.75, t_end=4000.0, **kw)
    b = dsm_mod.Ensemble(n_chains=n, seed=74, sync_dt=0.75, t_end=4000.0, lanes_per_chain=16, **kw)
    if small:
        a.set_schedule(small_slot=small, z_margin_sd=0.01)
    for x in (a, b):
        x.init_equilibrium()
    deferred = 0
    for t in (55.0, 56.0, 112.25):
        assert a.advance(t) == b.advance(t)
        deferred += a.window_stats()["deferred"]
    assert (deferred > 0) == (small > 0)
    a.advance_series(55.0, 2)
    for t in (167.25, 222.25):
        b.advance(t)
    if kw["eq_type"] != 0:
        ga, ca = a.gt_raw()
        gb, cb = b.gt_raw()
        assert np.array_equal(ca, cb)
        if small:  # a sum cut in two FP32 pieces where the chain changed its slot
            assert np.abs(ga - gb).max() <= 2.0**-22 * np.abs(gb).max()
        else:
            assert np.array_equal(ga, gb)
    assert_bitexact(gpu_state(a), gpu_state(b), what=f"slices {kw}")


def test_lockstep_abort_between_slices(dsm_mod):
    """A launch in time slices told to abort while it runs, then run to its end:
    no sample is lost (level-0 sums are cut in two FP32 pieces there)."""
    kw = dict(nk=300, beta=0.5, n_chains=6000, seed=75, eq_type=1, corr_p=64, corr_m=8, sync_dt=1.0, t_end=4000.0)
    a = dsm_mod.Ensemble(**kw)
    b = dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    flag = np.zeros(1, np.int32)

    def stop():
        flag[0] = 1
    timer = threading.Timer(0.1, stop)
    timer.start()
    a.advance(1500.0, abort=flag)
    timer.join()
    a.advance(1500.0)
    b.advance(1500.0)
    ga, ca = a.gt_raw()
    gb, cb = b.gt_raw()
    assert np.array_equal(ca, cb)
    assert np.abs(ga - gb).max() <= 2.0**-22 * np.abs(gb).max()
    assert_bitexact(gpu_state(a), gpu_state(b), what="abort between slices")


@pytest.mark.parametrize("n,lanes", [(N, 0), (64, 16), (64, 32)])
@pytest.mark.parametrize("q", [12.0, 15.0, 17.0, 40.0])
def test_exponents_beyond_the_short_form(dsm_mod, oracle_mod, n, lanes, q):
    """Strands so long that sliding exponents reach 54, 84, 108 and 600 (single
    Kuhn steps): below, near and above the limit of the short exponential, where the
    full rate pass takes over, with scales far below the start's."""
    kw = dict(nk=140, n_chains=n, seed=77, beta=0.5)
    g, o = dsm_mod.Ensemble(lanes_per_chain=lanes, **kw), oracle_mod.Oracle(**kw)
    g.init_equilibrium()
    heads, qn, tau = g.get_chains()
    rng = np.random.default_rng(5)
    for c in rng.choice(n, n // 4, replace=False):
        Z = int(heads["Z"][c])
        if Z > 6:
            s = int(rng.integers(2, Z - 2))
            qn[c, s, :3] = np.float32(q) * np.array([0.6, 0.0, 0.8], np.float32)
    g.set_chains(heads, qn, tau)
    o.set_state(heads["Z"], qn, tau, T=g.get_ext()["T"])
    for t in (0.05, 0.5):
        assert g.advance(t) == o.run(t)
    assert_bitexact(gpu_state(g), o.get_state(), what=f"|Q|={q}")
