"""One chain per warp for ensembles that are resident so (24 chains per SM), two per
warp beyond: the default schedule, batches, and the allocation-free step.  The state
and the sums do not depend on it."""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state
from test_zz_no_alloc import STATE_DTYPE, _bind

pytestmark = pytest.mark.gpu
KAP = (0.0, 2.0e-3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)
EDGE = 24 * 152


@pytest.mark.parametrize("n", [1, 33, EDGE, EDGE + 1])
@pytest.mark.parametrize("kw", [dict(eq_type=0), dict(eq_type=1, corr_p=16, corr_m=2),
                                dict(eq_type=2, corr_p=8, corr_m=2), dict(kappa=KAP)], ids=str)
def test_default_equals_two_per_warp(dsm_mod, n, kw):
    kw = dict(nk=40, n_chains=n, seed=91, sync_dt=0.5, t_end=100.0, **kw)
    a, b = dsm_mod.Ensemble(**kw), dsm_mod.Ensemble(lanes_per_chain=16, **kw)
    for x in (a, b):
        x.init_equilibrium()
    for t in (0.7, 3.0):
        assert a.advance(t) == b.advance(t)
    assert_bitexact(gpu_state(a), gpu_state(b), what=f"n={n}")
    if "kappa" in kw:
        sa, sb = a.stress(), b.stress()
        assert np.array_equal(sa[0], sb[0]) and sa[1] == sb[1]
    elif kw["eq_type"]:
        assert np.array_equal(a.gt_raw()[0], b.gt_raw()[0])
    if n > 1:  # the schedule the ensemble had before goes on from a request without lanes
        a.set_schedule(small_slot=30)
        assert a.schedule()[-2]["lanes"] == 16
        assert a.advance(4.0) == b.advance(4.0)
        assert_bitexact(gpu_state(a), gpu_state(b), what=f"n={n}, set_schedule")


@pytest.mark.parametrize("sizes", [(700, 900, 1100), (1500, 1500, 1500), (900, 5000)], ids=str)
@pytest.mark.parametrize("kappa", [(0.0,) * 9, KAP], ids=["eq", "shear"])
def test_batch_widths(dsm_mod, sizes, kappa):
    """Batches whose chains are together resident one per warp, are not, and a batch
    with an ensemble that is not by itself."""
    kws = [dict(nk=90 + 2 * i, n_chains=n, seed=92, stream=i, kappa=kappa) for i, n in enumerate(sizes)]
    a = [dsm_mod.Ensemble(**k) for k in kws]
    b = [dsm_mod.Ensemble(lanes_per_chain=32, **k) for k in kws]
    for x in a + b:
        x.init_equilibrium()
    ev = dsm_mod.advance_batch(a, 1.5)
    assert list(ev) == [x.advance(1.5) for x in b]
    for x, y in zip(a, b):
        assert_bitexact(gpu_state(x), gpu_state(y), what=f"batch {sizes}")


@pytest.mark.parametrize("kappa,nk,n", [((0.0,) * 9, 60, EDGE + 1), (KAP, 60, EDGE + 1), ((0.0,) * 9, 60, 14600),
                                        ((0.0,) * 9, 131, 7000), ((0.0,) * 9, 300, 4000)])
def test_noalloc_widths(dsm_mod, kappa, nk, n):
    import torch

    lib = _bind(dsm_mod)
    e = dsm_mod.Ensemble(nk=nk, n_chains=n, seed=93, kappa=kappa)
    e.init_equilibrium()
    heads, qn, tau = e.get_chains()
    ext = e.get_ext()
    st = np.zeros(n, STATE_DTYPE)
    st["Z"], st["scale"], st["hash"], st["nk"] = heads["Z"], ext["S"], ext["hash"], nk
    d = [torch.from_numpy(x).cuda() for x in (qn.copy(), tau.copy(), st.view(np.uint8).copy(), np.zeros(8 * n, np.float32))]
    ev = C.c_uint64(0)
    torch.cuda.synchronize()
    rc = lib.dsm_advance_noalloc(C.byref(e.params), *[C.c_void_p(x.data_ptr()) for x in d], 2.0, -1, None, C.byref(ev))
    assert rc == 0, lib.dsm_noalloc_last_error()
    torch.cuda.synchronize()
    assert ev.value == e.advance(2.0)
    got, x = d[2].cpu().numpy().view(STATE_DTYPE), e.get_ext()
    h, q, t = e.get_chains()
    assert np.array_equal(got["Z"], h["Z"]) and np.array_equal(got["hash"], x["hash"])
    assert np.array_equal(got["time_ticks"], x["T"])
    m = np.arange(nk)[None, :] < h["Z"][:, None]
    assert np.array_equal(d[0].cpu().numpy()[m].view(np.uint32), q[m].view(np.uint32))
