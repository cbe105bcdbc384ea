"""v2c_rsf_newton with its outputs in rows of the states (GPU): every state is
read before its outputs are written, as with separate arrays, so the results
are those, bit for bit."""
import ctypes

import numpy as np
import pytest

from oracle import bindings as B
from velo2cycles_gb300 import abi, mic, newton, synth
from velo2cycles_gb300._lib import call

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(built_lib, oracle_built):
    m = mic.from_case(synth.make_case("tiny", seed=3))
    S = newton.rsf_states(256, seed=1)
    ref, _, _ = B.rsf_newton(S, rtol=1e-10, maxit=200)
    newton.load(m, newton.random_params(3, B.rsf_features(S),
                                        np.stack([np.log(ref[abi.RO_V]), ref[abi.RO_PHI]], 1)))
    yield m
    m.close()


def _states(n):
    S = newton.rsf_states(n, seed=n)
    k = np.arange(n)
    S[abi.RS_TAUOLD, k % 97 == 3] = 1e-3   # far below the yield: the floor
    none = k % 131 == 5                    # no load at all: degenerate
    S[abi.RS_TAUOLD, none] = 0.0
    S[abi.RS_EDOT, none] = 0.0
    return S


# the first output row at state row 0, in the middle, at the end, and running
# past the states' end or up to their start
@pytest.mark.parametrize("row", [0, 5, abi.RS_N - abi.RO_N, abi.RS_N - 1, -3])
@pytest.mark.parametrize("guess", [abi.GUESS_PLAIN, abi.GUESS_LEARNED])
@pytest.mark.parametrize("precision", [abi.NEWTON_SPLIT, abi.NEWTON_FP64])
@pytest.mark.parametrize("n", [1, 4097])
def test_outputs_in_rows_of_the_states(ctx, n, precision, guess, row):
    import torch
    S = _states(n)
    ctx.set_params(newton_precision=precision)
    try:
        want, wit = newton.solve(ctx, S, guess)
        block = torch.zeros((abi.RS_N + 2 * abi.RO_N, n), dtype=torch.float64, device="cuda")
        states = block[abi.RO_N:abi.RO_N + abi.RS_N]
        states.copy_(torch.from_numpy(S))
        out = block[abi.RO_N + row:2 * abi.RO_N + row]
        it = torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.current_stream().synchronize()
        call("v2c_rsf_newton", ctx.h, ctypes.c_void_p(states.data_ptr()), n, int(guess),
             ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(it.data_ptr()))
        ctx.synchronize()
    finally:
        ctx.set_params(newton_precision=abi.NEWTON_SPLIT)
    assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(it.cpu().numpy(), wit)
    kept = [r for r in range(abi.RS_N) if not row <= r < row + abi.RO_N]
    assert np.array_equal(states.cpu().numpy()[kept], S[kept])
