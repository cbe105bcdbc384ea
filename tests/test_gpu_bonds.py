"""Replacing the boundary table (GPU): a refused table leaves the one in
force, for the Stokes matrix and for the boundary rows of marker2nodes, and
valid tables with more and with fewer rows take its place.  The matrix against
the restatement, bit for bit, as in test_gpu_stokes.py; marker2nodes against
its own result before the refused call."""
import numpy as np
import pytest

import oracle
from velo2cycles_gb300 import abi, mic
from velo2cycles_gb300._lib import V2CError

from .parity import M2N_OUT, stokes_case

pytestmark = pytest.mark.gpu


def _matrix(case, ctl):
    rc, ref = oracle.Restatement(case.copy()).stokes_assemble(**ctl)
    assert rc == 0
    return ref


def _same(got, ref):
    for k in ("ia", "ja", "a", "b"):
        assert np.array_equal(got[k], ref[k], equal_nan=k in ("a", "b")), k


def _refused(m, case, bondm, extra):
    """extra rows appended (or taken off), bondm refers past the end"""
    bn, bv = case.bondn.copy(), case.bondv.copy()
    if extra >= 0:
        bn, bv = np.append(bn, np.ones(3 * extra, bn.dtype)), np.append(bv, np.ones(4 * extra))
    else:
        bn, bv = bn[:3 * extra], bv[:4 * extra]
    with pytest.raises(V2CError) as e:
        m.set_bonds(bondm, bn, bv)
    assert e.value.code == abi.ERR_ARG


@pytest.mark.parametrize("name", ["tiny", "small"])
def test_refused_and_replaced_tables(built_lib, oracle_built, name):
    c, ctl = stokes_case(6, name=name)
    m = mic.from_case(c)
    ref = _matrix(c, ctl)
    _same(m.stokes_assemble(**ctl), ref)
    for extra in (0, 5000, -7):
        bad = c.bondm.copy()
        bad[[0, 5, -1]] = [c.bondnum + max(extra, 0), 1, -1]
        _refused(m, c, bad, extra)
        _same(m.stokes_assemble(**ctl), ref)
    # more rows: a copy of every row, with other constants, for half the unknowns
    more = c.copy()
    rows = c.bondnum
    more.bondn = np.concatenate([c.bondn, c.bondn])
    more.bondv = np.concatenate([c.bondv, c.bondv])
    more.bondv[4 * rows::4] += 2.5
    swap = (c.bondm > 0) & (np.arange(c.bondm.size) % 2 == 0)
    more.bondm[swap] += rows
    # fewer: no temperature rows, which are the last
    fewer = c.copy()
    fewer.bondm[3 * c.nodenum:] = 0
    left = int(fewer.bondm.max()) + 1
    fewer.bondn, fewer.bondv = c.bondn[:3 * left].copy(), c.bondv[:4 * left].copy()
    assert left < rows
    for case in (more, fewer, c):
        m.set_bonds(case.bondm, case.bondn, case.bondv)
        want = _matrix(case, ctl)
        assert case is c or case is fewer or not np.array_equal(want["b"], ref["b"])
        _same(m.stokes_assemble(**ctl), want)
        _refused(m, case, np.full(case.bondm.size, case.bondnum), 0)
        _same(m.stokes_assemble(**ctl), want)
    m.close()


def test_refused_table_and_boundary_rows(built_lib):
    c, _ = stokes_case(7, name="tiny")
    m = mic.from_case(c)
    m.marker2nodes()
    want = m.download_nodes(M2N_OUT)
    _refused(m, c, np.full(c.bondm.size, c.bondnum + 40), 3)
    m.upload_nodes(c.nodes)
    m.set_params(compressiblemode=1)  # the rows are built anew, twice
    m.marker2nodes()
    m.set_params(compressiblemode=0)
    m.upload_nodes(c.nodes)
    m.upload_markers(c.marks, c.markt)
    m.marker2nodes()
    got = m.download_nodes(M2N_OUT)
    for f in M2N_OUT:
        assert np.array_equal(got[f], want[f], equal_nan=True), abi.node_field_names()[f]
    m.close()
