"""Which ensembles the lockstep kernel runs, with how many lanes and time slices (the
bit-for-bit tests of that kernel hold only where it is the one that runs), and its
plans in the other ways to advance: batches, captured series, saved states, an
abort between two slices."""
import threading

import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu
N = 7400
TICKS = 2.0**32
SLICED = dict(nk=300, beta=0.5, n_chains=6000)


def gt(p, m, **kw):
    return dict(dict(eq_type=1, corr_p=p, corr_m=m, sync_dt=1.0, t_end=4000.0), **kw)


def same_run(a, b, times, what):
    for t in times:
        assert a.advance(t) == b.advance(t)
    assert_bitexact(gpu_state(a), gpu_state(b), what=what)


@pytest.mark.parametrize("kw,lanes", [
    (dict(nk=75, beta=4.0), 4), (dict(nk=90, beta=3.0), 4), (dict(nk=100), 4), (dict(nk=131), 4),
    (dict(nk=200, beta=0.5), 8), (dict(nk=463, beta=0.5), 8), (dict(nk=100, cd_flag=0), 4), (dict(nk=100, z_max=52), 4),
    (gt(16, 2, nk=151), 4), (gt(64, 8, nk=200), 4),
    (gt(96, 4, nk=240, beta=0.5), 8), (gt(8, 2, nk=175, eq_type=2), 4),
    (gt(64, 8, nk=300, sync_dt=0.25), 8), (gt(64, 8, nk=463, beta=0.5, sync_dt=0.1), 8), (gt(8, 2, nk=300, sync_dt=0.5, eq_type=2), 8)], ids=str)
def test_kernel_of_the_plan(dsm_mod, kw, lanes):
    k = dsm_mod.Ensemble(n_chains=N, seed=71, **kw).step_kernel()
    assert k["lockstep"] and k["lanes"] == lanes


@pytest.mark.parametrize("kw", [dict(nk=20), dict(nk=200, gex=(1.0, 1.0, 1000.0, 100.0)), dict(nk=500, beta=10.0), gt(64, 8, nk=200, beta=0.5), gt(64, 8, nk=150, beta=2.0),
                                gt(64, 8, nk=200, beta=4.0), gt(64, 8, nk=150, eq_type=2), gt(64, 8, nk=300, beta=0.25),
                                gt(64, 8, nk=200, sync_dt=0.25), gt(64, 8, nk=200, sync_dt=0.5, eq_type=2),
                                dict(nk=200, lanes_per_chain=16), dict(nk=200, lanes_per_chain=32),
                                dict(nk=200, kappa=(0.0, 2.0e-3) + (0.0,) * 7)], ids=str)
def test_tiles_otherwise(dsm_mod, kw):
    assert not dsm_mod.Ensemble(n_chains=N, seed=71, **kw).step_kernel()["lockstep"]
    assert not dsm_mod.Ensemble(n_chains=900, nk=200, seed=71).step_kernel()["lockstep"]


@pytest.mark.parametrize("kw", [gt(16, 2, nk=300, sync_dt=0.25), gt(64, 8, nk=200), gt(96, 4, nk=240, beta=0.5),
                                gt(64, 8, nk=300, sync_dt=0.5, eq_type=2), gt(8, 2, nk=175, eq_type=2)], ids=str)
def test_correlators(dsm_mod, kw):
    """G(t) and MSD sums of lockstep plans against 16-lane tiles, over windows that end
    inside, at and after full sample buffers (64 samples)."""
    a, b = dsm_mod.Ensemble(n_chains=N, seed=80, **kw), dsm_mod.Ensemble(n_chains=N, seed=80, lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    dt = kw["sync_dt"]
    for samples in (80, 100, 160, 192):
        t = samples * dt
        assert a.advance(t) == b.advance(t)
        assert a.step_kernel()["lockstep"]
        ga, ca = a.gt_raw()
        gb, cb = b.gt_raw()
        assert np.array_equal(ca, cb) and np.array_equal(ga, gb)
    assert_bitexact(gpu_state(a), gpu_state(b), what="correlator")
    assert np.array_equal(a.r1(), b.r1())


@pytest.mark.parametrize("kw", [dict(nk=131), dict(nk=200, beta=0.5), dict(nk=463, beta=0.5), dict(nk=90, beta=3.0),
                                dict(nk=100, cd_flag=0), dict(nk=100, z_max=52)], ids=str)
def test_against_the_oracle(dsm_mod, oracle_mod, kw):
    g, o = dsm_mod.Ensemble(n_chains=N, seed=87, **kw), oracle_mod.Oracle(n_chains=N, seed=87, **kw)
    g.init_equilibrium()
    o.init_equilibrium()
    assert g.advance(30.0) == o.run(30.0)
    assert g.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(g), o.get_state(), what=f"{kw}")


@pytest.mark.parametrize("q", [12.0, 15.0, 17.0, 40.0])
def test_exponents_beyond_the_short_form(dsm_mod, oracle_mod, q):
    """Strands so long that sliding exponents pass the limit of the short exponential."""
    kw = dict(nk=200, n_chains=N, seed=88, beta=0.5)
    g, o = dsm_mod.Ensemble(**kw), oracle_mod.Oracle(**kw)
    g.init_equilibrium()
    heads, qn, tau = g.get_chains()
    rng = np.random.default_rng(5)
    for c in rng.choice(N, N // 4, replace=False):
        qn[c, int(rng.integers(2, int(heads["Z"][c]) - 2)), :3] = np.float32(q) * np.array([0.6, 0.0, 0.8], np.float32)
    g.set_chains(heads, qn, tau)
    o.set_state(heads["Z"], qn, tau, T=g.get_ext()["T"])
    assert g.advance(20.0) == o.run(20.0)
    assert g.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(g), o.get_state(), what=f"|Q|={q}")


@pytest.mark.parametrize("kw", [dict(nk=100), gt(64, 8, nk=200), gt(64, 8, nk=200, eq_type=2), gt(64, 8, **SLICED),
                                dict(gt(16, 2, eq_type=2), **SLICED), dict(nk=100, z_max=52)], ids=str)
def test_short_and_long_windows(dsm_mod, kw):
    """A default lockstep ensemble runs tiles where a launch has few events per chain; the
    state, and what does not depend on where the windows end, are those of tiles."""
    kw = dict(dict(n_chains=N), **kw)
    a, b = dsm_mod.Ensemble(seed=89, **kw), dsm_mod.Ensemble(seed=89, lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    t = 0.0
    for dt, lock in ((0.25, False), (30.0, True), (0.5, False), (0.7, False), (40.0, True)):
        t += dt
        assert a.advance(t) == b.advance(t)
        assert a.step_kernel()["lockstep"] == lock
    for dt, n, lock in ((0.5, 4, False), (20.0, 2, True), (0.5, 4, False)):
        assert a.advance_series(dt, n)[0] == b.advance_series(dt, n)[0]
        assert a.step_kernel()["lockstep"] == lock
        t += dt * n
    for dt, lock in ((0.5, False), (30.0, True)):
        t += dt
        assert dsm_mod.advance_batch([a], t)[0] == b.advance(t)
        assert a.step_kernel()["lockstep"] == lock
    done = int(b.get_ext()["step"].mean())
    for limit, lock in ((done + 40, False), (done + 1500, True), (done + 1540, False)):
        assert a.advance(1.0e6, step_limit=limit) == b.advance(1.0e6, step_limit=limit)
        assert a.step_kernel()["lockstep"] == lock
    assert_bitexact(gpu_state(a), gpu_state(b), what="short and long windows")
    if "eq_type" in kw:
        assert np.array_equal(a.gt_raw()[0], b.gt_raw()[0]) and np.array_equal(a.gt_raw()[1], b.gt_raw()[1])
    # chains set anew begin at their own time, not at the handle's
    heads, qn, tau = a.get_chains()
    heads["time"] = 0.0
    for _ in range(2):
        for x in (a, b):
            x.set_chains(heads, qn, tau)
        for t, lock in ((30.0, True), (30.5, False), (70.5, True)):
            assert a.advance(t) == b.advance(t)
            assert a.step_kernel()["lockstep"] == lock
    assert_bitexact(gpu_state(a), gpu_state(b), what="chains set anew")


def test_slices_of_a_launch(dsm_mod):
    e = dsm_mod.Ensemble(seed=74, **SLICED)
    e.init_equilibrium()
    e.advance(55.0)
    assert e.step_kernel() == {"lockstep": True, "lanes": 8, "slot": e.step_kernel()["slot"], "slices": 4}
    e.advance(65.0)  # some 600 events per chain
    assert e.step_kernel()["lockstep"] and e.step_kernel()["slices"] == 1
    heads, qn, tau = e.get_chains()
    heads["time"] = 0.0
    e.set_chains(heads, qn, tau)
    e.advance(55.0)
    assert e.step_kernel()["slices"] == 4


@pytest.mark.parametrize("ends,slices", [((80.0, 81.0, 161.0), 1), ((80.0, 160.0, 240.0), 4)], ids=str)
def test_slices_of_a_series(dsm_mod, ends, slices):
    """The shortest window of a series decides: slices of a window of a few dozen events
    would load and store every chain for a handful of them."""
    a, b = (dsm_mod.Ensemble(seed=79, lanes_per_chain=k, **SLICED) for k in (0, 16))
    for x in (a, b):
        x.init_equilibrium()
    a.series_start(ends)
    while a.poll() is None:
        pass
    assert a.step_kernel()["lockstep"] and a.step_kernel()["slices"] == slices
    for t in ends:
        b.advance(t)
    assert_bitexact(gpu_state(a), gpu_state(b), what="series")


def test_batch_of_lockstep_ensembles(dsm_mod):
    """Two lockstep ensembles in one launch, beside groups of other kernels."""
    kws = [dict(gt(64, 8, nk=200), n_chains=N), dict(gt(64, 8, nk=160), n_chains=8000), dict(nk=170, n_chains=N),
           dict(gt(64, 8, nk=200), n_chains=900), dict(nk=30, n_chains=500)]
    a = [dsm_mod.Ensemble(seed=76, stream=i, **k) for i, k in enumerate(kws)]
    b = [dsm_mod.Ensemble(seed=76, stream=i, lanes_per_chain=16, **k) for i, k in enumerate(kws)]
    assert [x.step_kernel()["lockstep"] for x in a] == [True, True, True, False, False]
    for x in a + b:
        x.init_equilibrium()
    for t in (20.0, 45.0):
        ev = dsm_mod.advance_batch(a, t)
        assert list(ev) == [x.advance(t) for x in b]
        assert [x.step_kernel()["lockstep"] for x in a] == [True, True, True, False, False]
    for x, y in zip(a, b):
        assert_bitexact(gpu_state(x), gpu_state(y), what="batch")
    # (chains of the first outgrow the group's slot, which is the second's: their
    # level-0 sums are cut in two FP32 pieces there, in tiles as here)
    assert a[0].window_stats()["deferred"] > 0 == a[1].window_stats()["deferred"]
    assert np.array_equal(a[0].gt_raw()[1], b[0].gt_raw()[1])
    assert np.array_equal(a[1].gt_raw()[0], b[1].gt_raw()[0])


@pytest.mark.parametrize("z_max", [0, 52], ids=["classes", "captured"])
def test_series(dsm_mod, z_max):
    """An equilibrium series: size classes issue its windows, a plan of one launch
    replays them from a captured graph."""
    kw = dict(nk=100, z_max=z_max, n_chains=N, seed=77)
    a, b = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    assert a.step_kernel()["lockstep"] and (a.schedule() == []) == (z_max > 0)
    for x in (a, b):
        x.init_equilibrium()
    for _ in range(2):
        assert a.advance_series(20.0, 3)[0] == b.advance_series(20.0, 3)[0]
        assert a.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(a), gpu_state(b), what="series")


def test_saved_and_reloaded(dsm_mod, tmp_path):
    kw = dict(gt(64, 8, nk=200), n_chains=N, seed=78)
    a, b, c = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    a.init_equilibrium()
    a.advance(20.0)
    a.checkpoint(str(tmp_path / "k"))
    for x in (b, c):
        x.restore(str(tmp_path / "k"))
    assert b.step_kernel()["lockstep"]
    a.advance(45.0)
    same_run(b, c, [45.0], "restored")
    assert a.step_kernel()["lockstep"] and b.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(a), gpu_state(b), what="continued")
    assert np.array_equal(a.gt_raw()[0], b.gt_raw()[0]) and np.array_equal(b.gt_raw()[0], c.gt_raw()[0])
    a.save(str(tmp_path / "c"))
    for x in (b, c):
        x.load(str(tmp_path / "c"))
    same_run(b, c, [65.0], "loaded")


def test_abort_between_two_slices(dsm_mod):
    """Told to abort while some chains wait between two slices: they stopped at the end
    of one, and no sample is lost."""
    kw = dict(gt(64, 8, **SLICED), seed=75)
    a, b = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    begin, end = 300.0, 3300.0
    assert a.advance(begin) == b.advance(begin)
    a_window = a.last_window()["kernel_ms"] * 1.0e-3
    flag = np.zeros(1, np.int32)
    timer = threading.Timer(0.45 * a_window * (end - begin) / begin, lambda: flag.__setitem__(0, 1))
    timer.start()
    assert a.advance(end, abort=flag) == -1
    timer.join()
    k = a.step_kernel()["slices"]
    assert k > 1
    T = a.get_ext()["T"] / TICKS
    piece = (end - begin) / k
    done = np.floor((T - begin) / piece + 1e-9).astype(int)  # slices each chain has finished
    assert done.max() >= 1 and T.min() < end
    stopped = (done >= 1) & (done < k) & (T - begin - done * piece < 1.0)  # just past a slice's end
    assert stopped.sum() > 50
    assert a.advance(end) != -1
    b.advance(end)
    ga, ca = a.gt_raw()
    gb, cb = b.gt_raw()
    assert np.array_equal(ca, cb)
    # a sum cut in two FP32 compensated pieces where the abort fell
    assert np.abs(ga - gb).max() <= 2.0**-22 * np.abs(gb).max()
    assert_bitexact(gpu_state(a), gpu_state(b), what="abort between slices")


def plan(e):
    k = e.step_kernel()
    return k["lockstep"], k["lanes"], k["slot"], [(c["slot"], c["lanes"], c["grid"]) for c in e.schedule()]


@pytest.mark.parametrize("kw", [dict(gt(64, 8, nk=200), n_chains=N), dict(nk=300, n_chains=N), dict(gt(64, 8, **SLICED))],
                         ids=str)
def test_autotune(dsm_mod, kw):
    """The tuner tries the lockstep default and the tiles, keeps the default unless tiles
    are clearly faster (they are not here), changes no trajectory, and returns what
    set_schedule takes to make the same plan."""
    a, b = dsm_mod.Ensemble(seed=85, **kw), dsm_mod.Ensemble(seed=85, lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    start = plan(a)
    best = a.autotune(20.0)
    assert best["candidates"] > 2
    assert plan(a) == start
    for k in range(best["candidates"]):
        b.advance(20.0 * (k + 1))
    assert_bitexact(gpu_state(a), gpu_state(b), what="after autotune")
    a.set_schedule(small_slot=90 if kw["nk"] == 200 else 0, lanes=16)
    assert not a.step_kernel()["lockstep"]
    a.set_schedule(best["small_slot"], best["large_grid"], best["lanes"])
    assert plan(a) == start
    same_run(a, b, [20.0 * (best["candidates"] + 1)], "the tuner's choice again")


@pytest.mark.parametrize("kw", [dict(gt(64, 8, nk=200), n_chains=N), dict(nk=200, n_chains=N), dict(gt(64, 8, nk=100), n_chains=1500),
                                dict(nk=200, n_chains=1500)], ids=str)
def test_class_form_of_a_default_plan(dsm_mod, kw):
    """The carved form of lockstep and of small ensembles: the classes of their 16-lane
    tiles in one launch, and the default plan back."""
    a, b = dsm_mod.Ensemble(seed=86, **kw), dsm_mod.Ensemble(seed=86, lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    start = plan(a)
    a.set_class_form(1)
    assert a.class_form() == 1 and not a.step_kernel()["lockstep"] and a.schedule()[0]["lanes"] == 16
    same_run(a, b, [20.0], "carved")
    a.set_class_form(0)
    assert a.class_form() == 0 and plan(a) == start
    same_run(a, b, [40.0], "back")
