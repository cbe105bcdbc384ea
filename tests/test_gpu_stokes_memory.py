"""What the Stokes assembly keeps on the device between calls (GPU): at most
256 MiB, the boundary table included.  A grid of 8.7 M nodes, whose table alone
is larger (32 bytes a node), leaves the free memory as it was, and a second
call uploads the table again."""
import ctypes

import numpy as np
import pytest

from velo2cycles_gb300 import abi, mic, synth
from velo2cycles_gb300._lib import call

pytestmark = pytest.mark.gpu


def test_nothing_large_is_kept(built_lib):
    import torch
    xn, yn = 3000, 2900
    gx, gy = np.arange(xn) * 100.0, np.arange(yn) * 100.0
    p = synth.default_params(xnumx=xn, ynumy=yn, xsize=gx[-1], ysize=gy[-1], xstpx=100.0,
                             ystpy=100.0, timesum=0.0)
    m = mic.MarkerInCell(p, 0)
    m.set_grid(gx, gy)
    m.set_rock_table(synth.rock_table())
    # every unknown is given (row 1; before timebond, vx too): one coefficient a row
    m.set_bonds(np.ones(4 * m.nn, dtype=np.int64), np.zeros(6, dtype=np.int64),
                np.array([0, 0, 0, 0, 7.0, 0, 0, 0]))
    ctl = abi.StokesCtl(**dict(abi.STOKES_DEFAULTS, mukoef=1.0, dt=1e8))
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        nnz, b = ctypes.c_long(0), np.zeros(3 * m.nn)
        call("v2c_stokes_assemble", m.h, ctypes.byref(ctl), 0, None, None, None,
             b.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.byref(nnz))
        assert nnz.value == 3 * m.nn
        inner = b.reshape(xn, yn, 3)[1:-1, 1:-1]
        assert (inner == 7.0).all()
        # (the allocator's own blocks are 2 MiB)
        assert free - torch.cuda.mem_get_info()[0] <= (256 + 8) << 20
    m.close()
