"""Slides next to the chain ends in the lockstep kernel: chains of a few strands, on
which most slides change a strand count that the chain-end rates are then read
from by other lanes of the chain.  Against the oracle, bit for bit."""
import pytest

from helpers import assert_bitexact, gpu_state

pytestmark = pytest.mark.gpu
N = 7400  # more chains than the tiles hold at once: the lockstep kernel runs


@pytest.mark.parametrize("nk,beta", [(75, 4.0), (90, 3.0), (75, 2.0)])
def test_slides_next_to_chain_ends(dsm_mod, oracle_mod, nk, beta):
    kw = dict(nk=nk, beta=beta, n_chains=N, seed=171)
    g, o = dsm_mod.Ensemble(**kw), oracle_mod.Oracle(**kw)
    g.init_equilibrium()
    o.init_equilibrium()
    assert g.advance(50.0) == o.run(50.0)
    assert g.step_kernel()["lockstep"]
    assert_bitexact(gpu_state(g), o.get_state(), what=f"N_K={nk}, beta={beta}")
