"""The floor test of the per-marker Newton on nearly unstressed markers (GPU):
strain rates of 1e-20 to 1e-18 1/s, whose squares are subnormal in FP32, load
the markers over a long step to above or below the yield at the 1e-40 floor.
Against the oracle's FP64 Newton on the problems the step collects: both meet a
relative residual of 1e-10, which fixes a slip rate to the same order (here the
friction term is proportional to it), and a marker stores it in FP32, 2^-24 of
it or, below 1.2e-38, half of 2^-149."""
import numpy as np
import pytest

from oracle import bindings as B
from velo2cycles_gb300 import abi, mic, newton, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guess", [abi.GUESS_PLAIN, abi.GUESS_LEARNED])
@pytest.mark.parametrize("dt", [3e6, 3e7])
def test_small_strain_rates_load_the_markers(built_lib, oracle_built, dt, guess):
    # (a band as wide as the model: its friction parameters everywhere)
    case = synth.make_case("small", seed=2, fault_hw=60e3, timestep=dt)
    n = case.n
    rng = np.random.default_rng(int(dt))
    rate, angle = 10.0 ** rng.uniform(-20, -18, n), rng.uniform(0, 2 * np.pi, n)
    case.marks[abi.MF_EXX], case.marks[abi.MF_EXY] = rate * np.cos(angle), rate * np.sin(angle)
    case.marks[abi.MF_XX][:] = 0.0
    case.marks[abi.MF_XY] = 10.0 ** rng.uniform(-5, -3, n)
    case.marks[abi.MF_PHI] = rng.uniform(4, 20, n)
    # the previous slip rates, all different, tell the collected problems apart
    case.marks[abi.MF_SLIPV] = 1e-12 * (1.0 + np.arange(n) / 4096.0)
    m = mic.from_case(case)
    S = newton.collect_states(m).cpu().numpy()
    at = np.rint((S[abi.RS_VOLD] / 1e-12 - 1.0) * 4096.0).astype(int)
    assert at.size > n // 2 and np.unique(at).size == at.size
    ref, _, nc = B.rsf_newton(S, rtol=1e-10, maxit=200)
    unloaded = S.copy()
    unloaded[abi.RS_EDOT] = 0.0
    ref0, _, _ = B.rsf_newton(unloaded, rtol=1e-10, maxit=200)
    want = ref[abi.RO_V]
    assert nc == 0
    # loads of rates below 1e-19 decide here, and both answers occur
    decided = (want > 1.1e-40) & (ref0[abi.RO_V] <= 1e-40) & (S[abi.RS_EDOT] < 1e-19)
    assert decided.sum() > 100 and (want == 1e-40).sum() > 100
    if guess == abi.GUESS_LEARNED:
        newton.load(m, newton.random_params(3))
    m.set_params(newton_guess=guess)
    m.marker2nodes()
    st = m.status()
    assert st["newton_nonconv"] == 0
    got = m.download_markers([abi.MF_SLIPV])[abi.MF_SLIPV][at]
    assert np.all(np.abs(got - want) <= 1e-6 * want + 2.0 ** -149)
    m.close()
