"""Flow rates out of the range of the short forms (exponents of 88 and more, scales
far below the start's) against the oracle, in both tile widths."""
import numpy as np
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [16, 32])
@pytest.mark.parametrize("q", [12.0, 15.0, 17.0, 40.0, 400.0])
def test_long_strands(dsm_mod, oracle_mod, lanes, q):
    kw = dict(nk=70, n_chains=96, seed=97, kappa=(0.0, 2.0e-3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0))
    g, o = dsm_mod.Ensemble(lanes_per_chain=lanes, **kw), oracle_mod.Oracle(**kw)
    g.init_equilibrium()
    heads, qn, tau = g.get_chains()
    rng = np.random.default_rng(6)
    for c in range(0, 96, 3):
        Z = int(heads["Z"][c])
        if Z > 6:
            qn[c, int(rng.integers(2, Z - 2)), :3] = np.float32(q) * np.array([0.6, 0.0, 0.8], np.float32)
    g.set_chains(heads, qn, tau)
    o.set_state(heads["Z"], qn, tau, T=g.get_ext()["T"])
    for t in (0.05, 0.6):
        assert g.advance(t) == o.run(t)
    assert_bitexact(gpu_state(g), o.get_state(), what=f"|Q|={q}")
