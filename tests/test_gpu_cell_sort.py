"""The allocation-free cell sort where its warps' groups of cells, its paired
half-warps and its bit-pattern bisection can go wrong (GPU): cells of 0 to
300 markers in random array order, cell counts that are no multiple of a
group, markers on the lines, outside the model, at zeros of both signs and on
lines below zero, lines closer than their upper words tell apart.  Against numpy's search and stable sort; integer results,
equal."""
import numpy as np
import pytest

from velo2cycles_gb300 import cellsort

pytestmark = pytest.mark.gpu

SHAPES = [
    (2, 2, [5], 0.0),              # one cell
    (2, 10, [0, 16, 17], 0.0),     # nine cells: a group and one more
    (5, 6, [15, 16], -1.5),        # pairs of half-warps, lines below zero
    (12, 8, [0, 1, 16, 17, 31, 32, 33], 0.0),
    (9, 14, [3, 64, 65, 300], -2.0),
    (40, 31, [0, 2, 16, 20], 0.0),
    (4, 5, [0, 1022, 1023, 1024, 2500], 0.0),  # slots past the ten bits
    (6200, 3, [0, 1, 2], 0.0),     # more lines than shared memory takes
]


@pytest.mark.parametrize("xn,yn,fill,x0", SHAPES)
def test_cells_and_order(built_lib, xn, yn, fill, x0):
    import torch
    rng = np.random.default_rng(xn * 100 + yn)
    gx = x0 + np.concatenate([[0.0], np.cumsum(rng.uniform(0.1, 2.0, xn - 1))])
    gy = x0 + np.concatenate([[0.0], np.cumsum(rng.uniform(0.1, 2.0, yn - 1))])
    if xn == 40:
        gx = 1000.0 + np.arange(xn) * 2.0 ** -25
    count = rng.choice(fill, size=(xn - 1) * (yn - 1))
    c = np.repeat(np.arange(count.size), count)
    c = rng.permutation(c)
    ix, iy = c // (yn - 1), c % (yn - 1)
    x = gx[ix] + rng.random(c.size) * (gx[ix + 1] - gx[ix])
    y = gy[iy] + rng.random(c.size) * (gy[iy + 1] - gy[iy])
    if c.size >= 16:
        x[0], y[1] = gx[-1], gy[-1]              # on the last lines
        x[2], y[3] = gx[0], gy[0]                # on the first
        x[4], y[5] = gx[0] - 3.0, gy[-1] + 3.0   # outside
        x[6], x[7], y[8] = -0.0, 0.0, -0.0
        k = xn // 2
        x[9], x[10] = gx[k], np.nextafter(gx[k], -np.inf)
    want = (np.clip(np.searchsorted(gx, x, side="right") - 1, 0, xn - 2) * (yn - 1) +
            np.clip(np.searchsorted(gy, y, side="right") - 1, 0, yn - 2))
    start = np.concatenate([[0], np.cumsum(np.bincount(want, minlength=count.size))])
    dev = torch.device("cuda:0")
    put = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
    new = lambda n: torch.full((n,), -7, dtype=torch.int32, device=dev)
    cell, perm, st = new(c.size), new(c.size), new(count.size + 1)
    cellsort.sort_cells_static(put(gx), put(gy), put(x), put(y), cell, perm, st)
    assert np.array_equal(cell.cpu().numpy(), want)
    assert np.array_equal(st.cpu().numpy(), start)
    assert np.array_equal(perm.cpu().numpy(), np.argsort(want, kind="stable"))
