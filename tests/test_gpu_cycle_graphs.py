"""Captured cycle steps after something they hold has changed (GPU): another
boundary table, another number of markers, another rock table, a network that
arrives, parameters that go and come back -- the graph steps give the eager
ones bit for bit throughout."""
import numpy as np
import pytest

from velo2cycles_gb300 import abi, cycle, mic, newton, synth

pytestmark = pytest.mark.gpu

NODES = [abi.NF_SXY, abi.NF_SXX, abi.NF_PHIS, abi.NF_TK, abi.NF_MVX, abi.NF_MVY, abi.NF_SPPE,
         abi.NF_NU, abi.NF_RK_SLIPRS_FINAL]
MARKS = [abi.MF_X, abi.MF_Y, abi.MF_XX, abi.MF_XY, abi.MF_PHI, abi.MF_SLIPV]


def _table(case, shift):
    """the case's boundary table with other constants and one more row"""
    bn = np.append(case.bondn, [0, 0, 0])
    bv = np.append(case.bondv, [0.0, 0.0, 0.0, 0.0])
    bv[0::4] *= 1.0 + shift
    bm = case.bondm.copy()
    on = np.flatnonzero(bm[3 * case.nodenum:])[::2] + 3 * case.nodenum
    bm[on] = case.bondnum
    bv[4 * case.bondnum] = 400.0 + shift
    return bm, bn, bv


def _fewer(case, n):
    return {f: v[:n] for f, v in case.marks.items()}, case.markt[:n]


@pytest.mark.parametrize("params", [{}, dict(interpolationmod=1, antidiffinter=1)])
def test_what_a_graph_holds_changes(built_lib, params):
    case = synth.make_case("tiny", seed=5, newton_guess=abi.GUESS_LEARNED, **params)
    fields = cycle.pulse_fields(case, cycle.Schedule())
    runs = []
    for graph in (False, True):
        m = mic.from_case(case)
        m.cycle_set_velocity(0, *fields[0])
        seen = []

        def steps(n=case.n):
            # from the same state, so that only the change tells stages apart
            m.upload_nodes(case.nodes)
            m.upload_markers(*_fewer(case, n))
            for _ in range(4):
                m.cycle_step(0, 1e8, use_graph=graph)
            n, mk = m.download_nodes(NODES), m.download_markers(MARKS)
            seen.append([n[f] for f in NODES] + [mk[f] for f in MARKS] + [m.cycle_slip()])

        steps()
        m.set_bonds(*_table(case, 0.5))
        steps()
        for n in (case.n - 777, case.n):
            steps(n)
        newton.load(m, newton.random_params(5))
        steps()
        rt = case.rt.copy()
        rt[abi.RT_GG, 2] *= 3.0
        m.set_rock_table(rt)
        steps()
        # rows built for other parameters, and again for these
        for mode in (1, 0, 1, 0):
            m.set_params(compressiblemode=mode)
            steps()
        m.set_bonds(case.bondm, case.bondn, case.bondv)
        steps()
        runs.append(seen)
        m.close()
    assert not np.array_equal(runs[0][0][3], runs[0][1][3])  # the new rows show
    for eager, graph in zip(*runs):
        for a, b in zip(eager, graph):
            assert np.array_equal(a, b, equal_nan=True)


def test_calls_after_a_replayed_step(built_lib):
    """What the host knows of the node fields after a step is the same when
    the step was replayed: marker2nodes has written the temperature, so the
    one uploaded in FP64 is no longer it, and the stress changes are kept."""
    case = synth.make_case("tiny", seed=5)
    fields = cycle.pulse_fields(case, cycle.Schedule())
    tk2 = case.nodes[abi.NF_TK] + 3.0
    got = []
    for graph in (False, True):
        m = mic.from_case(case)
        m.cycle_set_velocity(0, *fields[0])
        for _ in range(3):
            m.cycle_step(0, 1e8, use_graph=graph)
        m.upload_nodes({abi.NF_TK: case.nodes[abi.NF_TK] + 50.0, abi.NF_TK2: tk2})
        m.cycle_step(0, 1e8, use_graph=graph)
        m.interpolate_center2basic(1e8)
        m.marker_temperature()
        mk = m.download_markers([abi.MF_K])[abi.MF_K]
        got.append([mk] + list(m.download_nodes([abi.NF_EXXPL, abi.NF_EXXEL, abi.NF_TK]).values()))
        m.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)
