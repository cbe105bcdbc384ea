"""The tile sweeps at the edges of their tiles, strips and chunks (GPU):
node-row counts around the 32 rows of a tile and node columns around a strip,
cells that hold none, a few or hundreds of markers (column segments that do
not fit one staged chunk), markers on the exact halves and lines of their
cells, density per marker.  Against the oracle at the tolerance of
test_gpu_mic.py: an FP32 result of compensated sums, 1e-6 per entry."""
import numpy as np
import pytest

from velo2cycles_gb300 import abi, mic, synth

from .parity import (M2N_OUT, N2M_MARK, N2M_OUT, marker_errors, n2m_floors, node_errors,
                     oracle_for, over)

pytestmark = pytest.mark.gpu


def sweep_case(xn, yn, fill, seed=3, **kw):
    """A window of the large configuration with the markers per cell drawn
    from `fill`, some of them on exact halves and lines."""
    case = synth.make_case("c4", seed=seed, window=(1500, 100, xn, yn),
                           n_markers=(xn - 1) * (yn - 1) * max(fill), **kw)
    rng = np.random.default_rng(seed)
    ncy, per = yn - 1, max(fill)
    n = case.n
    # markers come 20 to a cell, cell by cell, over and over: deal them out
    # again, `per` candidates per cell
    cell = np.arange(n) // per
    ix, iy = cell // ncy, cell % ncy
    u, v = rng.random(n), rng.random(n)
    snap = rng.random(n)
    u[snap < 0.02] = 0.5
    v[(snap > 0.01) & (snap < 0.03)] = 0.5
    u[(snap > 0.03) & (snap < 0.04)] = 0.0
    v[(snap > 0.04) & (snap < 0.05)] = 0.0
    case.marks[abi.MF_X] = case.gx[ix] + u * (case.gx[ix + 1] - case.gx[ix])
    case.marks[abi.MF_Y] = case.gy[iy] + v * (case.gy[iy + 1] - case.gy[iy])
    count = rng.choice(fill, size=(xn - 1) * ncy)
    keep = np.arange(n) % per < count[cell]
    for f in case.marks:
        case.marks[f] = case.marks[f][keep]
    case.markt = case.markt[keep]
    return case


SHAPES = [
    (4, 4, [20], {}),               # the smallest grid
    (5, 32, [20], {}),              # yn - 1 = 31 cell rows: one tile, not full
    (18, 33, [16], {}),             # 33 node rows: a second tile of one row
    (17, 34, [0, 20], {}),          # empty cells
    (34, 65, [0, 1, 2, 40], {}),    # a third tile of one row, uneven cells
    (9, 40, [30], {}),              # 990 markers per segment: two chunks
    (6, 36, [0, 5, 300], {}),       # several chunks, a cell across chunks
    (19, 47, [9, 25], dict(densimod=1)),
    (70, 12, [3, 20], dict(antidiffinter=0)),
]


@pytest.mark.parametrize("xn,yn,fill,kw", SHAPES)
def test_scatter_and_gather_edges(built_lib, oracle_built, xn, yn, fill, kw):
    case = sweep_case(xn, yn, fill, **kw)
    m = mic.from_case(case)
    ref = oracle_for(case)
    m.marker2nodes()
    ref.marker2nodes()
    bad = over(node_errors(m.download_nodes(M2N_OUT), ref.nodes, M2N_OUT))
    assert not bad, bad
    floors = n2m_floors(ref)
    m.nodes2markers()
    ref.nodes2markers()
    bad = over(node_errors(m.download_nodes(N2M_OUT), ref.nodes, N2M_OUT))
    assert not bad, bad
    bad = over(marker_errors(m.download_markers(N2M_MARK), ref.marks, N2M_MARK, floors))
    assert not bad, bad
    m.close()


@pytest.mark.parametrize("mode", [1, 2])
def test_markers_at_the_model_edges(built_lib, oracle_built, mode):
    """Markers on, inside and outside the model's edges by distances on both
    sides of what an FP32 position resolves: only those strictly inside
    count (FP64 decides where FP32 cannot)."""
    case = synth.make_case("c1", seed=4, window=(0, 0, 12, 9), interpolationmod=mode)
    x, y = case.marks[abi.MF_X], case.marks[abi.MF_Y]
    xs, ys = case.gx[-1], case.gy[-1]
    d = np.array([0.0, 1e-9, 1e-4, 1e-2, 0.3, 3.0, 30.0])
    d = np.concatenate([d, -d[1:]])
    rng = np.random.default_rng(1)
    at = rng.permutation(case.n)[:8 * d.size].reshape(8, d.size)
    for k, (p, edge, sign) in enumerate([(x, 0.0, 1), (x, xs, -1), (y, 0.0, 1), (y, ys, -1)] * 2):
        p[at[k]] = edge + sign * d
    m = mic.from_case(case)
    ref = oracle_for(case)
    m.marker2nodes()
    ref.marker2nodes()
    bad = over(node_errors(m.download_nodes(M2N_OUT), ref.nodes, M2N_OUT))
    assert not bad, bad
    m.close()
