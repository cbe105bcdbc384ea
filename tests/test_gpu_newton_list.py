"""The FP64 phase of the state Newton with more states than its list holds
(2^18), left to it in every way (GPU): with a tolerance that the float-float
phase does not reach, ordinary states as an iterate and its iterations, some
loads degenerate, some states restarted from the plain start -- results and
iteration counts as in calls that fit the list, bit for bit."""
import numpy as np
import pytest

from oracle import bindings as B
from velo2cycles_gb300 import abi, mic, newton, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guess", [abi.GUESS_PLAIN, abi.GUESS_LEARNED])
def test_states_past_the_list(built_lib, oracle_built, guess):
    m = mic.from_case(synth.make_case("tiny", seed=3))
    T = newton.rsf_states(256, seed=1)
    ref, _, _ = B.rsf_newton(T, rtol=1e-10, maxit=200)
    newton.load(m, newton.random_params(3, B.rsf_features(T),
                                        np.stack([np.log(ref[abi.RO_V]), ref[abi.RO_PHI]], 1)))
    n = 400_003
    S = newton.rsf_states(n, seed=7)
    k = np.arange(n)
    S[abi.RS_TAUOLD, k % 97 == 3] = 1e-3   # the floor
    none = k % 13 == 5                     # degenerate
    S[abi.RS_TAUOLD, none] = 0.0
    S[abi.RS_EDOT, none] = 0.0
    # a tolerance of a few FP64 roundings: some states never meet it
    m.set_params(newton_rtol=1e-15, newton_maxit=30)
    before = m.status()
    out, it = newton.solve(m, S, guess)
    after = m.status()
    ordinary = ~none & (k % 97 != 3)
    assert (it[none] == 0).all() and (np.abs(it[ordinary]) > 4).sum() > (1 << 18)
    assert (it < 0).any() and (it[ordinary] > 0).any()
    if guess == abi.GUESS_LEARNED:
        assert after["newton_fallbacks"] > before["newton_fallbacks"]
    for part in np.array_split(k, 5):
        want, wit = newton.solve(m, S[:, part], guess)
        assert np.array_equal(out[:, part], want, equal_nan=True)
        assert np.array_equal(it[part], wit)
    m.close()
