"""The split Newton on state arrays, solved in phases (GPU).

* a state's results do not depend on where it lies in the call: block edges
  of the phases, the gathering of the states left to FP64, floors and
  degenerate loads among ordinary states, both starts -- bit for bit against
  the same states in another order;
* against the oracle's FP64 Newton at the tolerance of test_gpu_newton.py
  (both stop at a relative residual of 1e-10; slip rates within 1e-8);
* the conversions between FP64 and float pairs by bit pattern equal the
  rounded ones exactly, at ties, carries, the ends of their range, zeros,
  subnormals, infinities and NaN.
"""
import os
import subprocess

import numpy as np
import pytest

from oracle import bindings as B
from velo2cycles_gb300 import abi, build, mic, newton, synth

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def ctx(built_lib, oracle_built):
    m = mic.from_case(synth.make_case("tiny", seed=3))
    S = newton.rsf_states(256, seed=1)
    ref, _, _ = B.rsf_newton(S, rtol=1e-10, maxit=200)
    X = B.rsf_features(S)
    newton.load(m, newton.random_params(3, X, np.stack([np.log(ref[abi.RO_V]),
                                                        ref[abi.RO_PHI]], 1)))
    yield m
    m.close()


def _states(n):
    S = newton.rsf_states(n, seed=n)
    k = np.arange(n)
    S[abi.RS_TAUOLD, k % 97 == 3] = 1e-3   # far below the yield: the floor
    none = k % 131 == 5                    # no load at all: degenerate
    S[abi.RS_TAUOLD, none] = 0.0
    S[abi.RS_EDOT, none] = 0.0
    S[abi.RS_VOLD, k % 61 == 7] = 0.0      # no previous slip rate
    return S


@pytest.mark.parametrize("guess", [abi.GUESS_PLAIN, abi.GUESS_LEARNED])
@pytest.mark.parametrize("n", [1, 127, 129, 4095, 4097, 9001])
def test_phases(ctx, n, guess):
    S = _states(n)
    out, it = newton.solve(ctx, S, guess)
    order = np.random.default_rng(n).permutation(n)
    out2, it2 = newton.solve(ctx, S[:, order], guess)
    assert np.array_equal(out[:, order], out2) and np.array_equal(it[order], it2)
    assert (it >= 0).all()
    ref, _, nc = B.rsf_newton(S, rtol=1e-10, maxit=200)
    assert nc == 0
    live = ref[abi.RO_V] > 1e-40
    assert np.array_equal(out[abi.RO_V] > 1e-40, live)
    if live.any():
        rel = np.abs(out[abi.RO_V] / ref[abi.RO_V] - 1)[live]
        assert np.quantile(rel, 0.999) < 1e-8
        assert B.rsf_residual(S[:, live], out[abi.RO_V][live]).max() <= 1e-10


def test_more_states_left_than_the_list_holds(ctx):
    """270 000 degenerate loads among ordinary states: the FP64 phase's list
    (2^18) runs over, and nothing changes."""
    n = 270_003
    S = newton.rsf_states(n, seed=5)
    some = np.arange(n) % 90 == 1
    S[abi.RS_TAUOLD, ~some] = 0.0
    S[abi.RS_EDOT, ~some] = 0.0
    out, it = newton.solve(ctx, S, abi.GUESS_PLAIN)
    assert (out[abi.RO_V, ~some] == 1e-40).all() and (it[~some] == 0).all()
    want, wit = newton.solve(ctx, S[:, some], abi.GUESS_PLAIN)
    assert np.array_equal(out[:, some], want) and np.array_equal(it[some], wit)


def test_conversions_by_bit_pattern(tmp_path):
    rng = np.random.default_rng(2)
    x = [np.exp(rng.uniform(-100, 88, 100000)) * rng.choice([-1, 1], 100000)]
    one = 1.0 + np.arange(64) * 2.0 ** -23
    for d in (0.0, 2.0 ** -24, 2.0 ** -24 + 2.0 ** -52, 2.0 ** -24 - 2.0 ** -52, 2.0 ** -52,
              2.0 ** -23 - 2.0 ** -52):
        x += [one + d, -(one + d)]
    x.append(np.nextafter(2.0 ** np.arange(-160.0, 130.0), 0.0))     # carries
    x.append(2.0 ** np.arange(-160.0, 130.0) * (1 + 2.0 ** -52))
    x.append(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 3.4028235e38,
                       3.4028236e38, 1e300]))
    x = np.concatenate(x)
    exe, fin, fout = (str(tmp_path / f) for f in ("check", "in.bin", "out.bin"))
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", build.ARCH, "-o", exe,
                    os.path.join(HERE, "ff_bits_check.cu")], check=True)
    with open(fin, "wb") as f:
        np.array([x.size], np.int64).tofile(f)
        x.tofile(f)
    subprocess.run([exe, fin, fout], check=True)
    with open(fout, "rb") as f:
        got = np.fromfile(f, np.float32, 2 * x.size).reshape(-1, 2)
        wide = np.fromfile(f, np.float64, x.size)
    with np.errstate(all="ignore"):
        hi = x.astype(np.float32)
        lo = (x - hi.astype(np.float64)).astype(np.float32)
    for a, b in ((got[:, 0], hi), (got[:, 1], lo), (wide, hi.astype(np.float64))):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        bits = np.int64 if a.itemsize == 8 else np.int32
        assert ((a.view(bits) == b.view(bits)) | (np.isnan(a) & np.isnan(b))).all()
