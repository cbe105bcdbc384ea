"""The Stokes assembly's kept state (GPU): repeated assemblies give the same
arrays, and a new boundary table replaces the one on the device.  Against the
restatement, bit for bit, as in test_gpu_stokes.py."""
import numpy as np
import pytest

import oracle
from velo2cycles_gb300 import mic

from .parity import stokes_case

pytestmark = pytest.mark.gpu


def _same(got, ref):
    for k in ("ia", "ja", "a", "b"):
        assert np.array_equal(got[k], ref[k], equal_nan=k in ("a", "b")), k


@pytest.mark.parametrize("name", ["tiny", "small"])
def test_repeated_and_after_new_bonds(built_lib, oracle_built, name):
    c, ctl = stokes_case(5, name=name)
    m = mic.from_case(c)
    rc, ref = oracle.Restatement(c.copy()).stokes_assemble(**ctl)
    assert rc == 0
    _same(m.stokes_assemble(**ctl), ref)
    _same(m.stokes_assemble(**ctl), ref)
    # other boundary values and coefficients
    c2 = c.copy()
    c2.bondv = c.bondv.copy()
    c2.bondv[0::4] += 1.5
    c2.bondv[1::4] *= 0.5
    m.set_bonds(c2.bondm, c2.bondn, c2.bondv)
    rc, ref2 = oracle.Restatement(c2.copy()).stokes_assemble(**ctl)
    assert rc == 0 and not np.array_equal(ref2["b"], ref["b"])
    _same(m.stokes_assemble(**ctl), ref2)
    m.close()
