"""Transfers by kernels and by copies (GPU): pinned arrays of every kind the
batched calls accept, pageable ones and mixtures give the same values, FP64 ->
FP32 -> FP64 exactly, and the FP64 copies of the velocities and temperatures
follow either way; marker fields come in the host's numbering either way."""
import numpy as np
import pytest

from velo2cycles_gb300 import abi, mic, synth

pytestmark = pytest.mark.gpu

FIELDS = [abi.NF_VX, abi.NF_VY, abi.NF_PR, abi.NF_TK, abi.NF_TK2, abi.NF_SXX]


def _arrays(kind, values):
    import torch
    out = {}
    for k, f in enumerate(FIELDS):
        pinned = kind == "pinned" or kind == "offset" or (kind == "mixed" and k % 2 == 0)
        pad = 3 if kind == "offset" else 0  # a view that starts inside its allocation
        t = torch.zeros(values[f].size + pad, dtype=torch.float64, pin_memory=pinned)
        out[f] = t.numpy()[pad:]
        out[f][:] = values[f]
    return out


@pytest.mark.parametrize("window", [(0, 0, 5, 5), (3, 2, 37, 29)])
@pytest.mark.parametrize("kind", ["pinned", "offset", "pageable", "mixed"])
def test_batched_transfers(built_lib, kind, window):
    case = synth.make_case("c1", seed=4, window=window)
    m = mic.from_case(case)
    rng = np.random.default_rng(1)
    up = {f: rng.normal(1.0, 0.5, m.nn) for f in FIELDS}
    m.upload_nodes(_arrays(kind, up))
    want = {f: up[f].astype(np.float32).astype(np.float64) for f in FIELDS}
    zero = {f: np.zeros(m.nn) for f in FIELDS}
    got = _arrays(kind, zero)
    m.download_nodes(list(got), into=got)
    late = _arrays(kind, zero)
    m.download_nodes_async(late)
    m.upload_nodes(_arrays(kind, {f: -up[f] for f in FIELDS}))  # after the snapshot
    m.wait_downloads()
    for f in FIELDS:
        assert np.array_equal(got[f], want[f])
        assert np.array_equal(late[f], want[f])
    # strain rates from the kept FP64 velocities: of the second upload
    m.recompute_stress_strainrate(1e8)
    exx = m.download_node(abi.NF_EXX)
    yn = case.gy.size
    vx, vy = -up[abi.NF_VX], -up[abi.NF_VY]
    k = 1 * yn + 1
    ref = 0.5 * ((vx[k - 1] - vx[k - yn - 1]) / (case.gx[1] - case.gx[0]) -
                 (vy[k - yn] - vy[k - yn - 1]) / (case.gy[1] - case.gy[0]))
    assert abs(exx[k] - ref) <= 2.0 ** -23 * abs(ref)
    m.close()


@pytest.mark.parametrize("n", [1, 255, 4001])
@pytest.mark.parametrize("kind", ["pinned", "offset", "mixed"])
def test_marker_download(built_lib, kind, n):
    import torch
    case = synth.make_case("c1", seed=4, window=(3, 2, 37, 29))
    order = np.random.default_rng(2).permutation(case.n)[:n]  # no cell order
    for f in case.marks:
        case.marks[f] = case.marks[f][order]
    case.markt = case.markt[order]
    m = mic.from_case(case)
    m.marker2nodes()
    m.nodes2markers_move()
    fields = [abi.MF_X, abi.MF_Y, abi.MF_K, abi.MF_XX, abi.MF_PHI, abi.MF_VX]
    want = m.download_markers(fields)
    into = {}
    for k, f in enumerate(fields):
        pad = 3 if kind == "offset" else 0
        t = torch.full((n + pad,), -7.0, dtype=torch.float64,
                       pin_memory=kind != "mixed" or k % 2 == 0)
        into[f] = t.numpy()[pad:]
    got = m.download_markers(fields, into=dict(into))
    for f in fields + ["markt"]:
        assert np.array_equal(got[f], want[f]), f
    assert np.array_equal(into[abi.MF_X], want[abi.MF_X])  # in place
    m.close()
