"""Plans over format arrays that are the caller's own (b200spmm_plan_create_device): what the converter would not have
made is either refused or multiplied as it stands, by every kernel that may take it."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
import parity
from cases import dense_b
from hopper_spmm_b200 import _capi as capi

pytestmark = pytest.mark.gpu

ROWS, COLS, PAD = 715, 1037, 0xFFFFFFFF
DENSITY = {"units": 0.01, "tiles": 0.3}  # row units; tiles, and the narrow format (rows of 300 entries) beside them


def matrix(kind, dt):
    rng = np.random.default_rng(3)
    mask = rng.random((ROWS, COLS)) < DENSITY[kind]
    mask[:, 128:192] |= kind == "tiles"  # tiles of neighbouring columns, which may come as boxes
    mask[200:240] = False
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.uint32)
    ci = np.nonzero(mask)[1].astype(np.uint32)
    return rp, ci, rng.uniform(0.1, 1, ci.size).astype(np.float32).astype(dt)


def arrays(rp, ci, v):
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(ROWS, COLS, rp, ci, v))
    info = capi.BtcfInfo()
    for k in ("rows", "cols", "nnzs", "total_row_windows", "eff_row_windows", "total_tiles", "row_window", "col_window"):
        setattr(info, k, getattr(f, k))
    info.dtype, info.elt_size = (capi.F16, 2) if v.dtype == np.float16 else (capi.TF32, 4)
    return info, {k: np.array(getattr(f, k)) for k in ("rowOffset", "tcA2B", "data", "rowIdx")}


def make_plan(info, a):
    import torch
    dev = {k: torch.from_numpy(a[k].view(np.int32) if a[k].dtype == np.uint32 else a[k]).cuda() for k in a}
    return hs.SpmmPlan(device_arrays=(info, dev["rowOffset"], dev["tcA2B"], dev["data"], dev["rowIdx"]))


def check(info, a, rp, ci, v, n, plain):
    import torch
    B = dense_b(info.cols, n, 9, v.dtype)
    plan = make_plan(info, a)
    try:
        C_out = torch.full((info.rows, n), float("nan"), device="cuda")
        plan.spmm(torch.from_numpy(B).cuda(), C_out)
        assert plan.launch_info().row_window == 16 or not plain
        parity.check(C_out.cpu().numpy(), info.rows, rp, ci, v, B)
    finally:
        plan.close()


def inside(rp, ci, v, rows, cols):
    """The part of the matrix in its first rows and columns."""
    r = np.repeat(np.arange(ROWS), np.diff(rp.astype(np.int64)))
    keep = (r < rows) & (ci < cols)
    return np.concatenate([[0], np.cumsum(np.bincount(r[keep], minlength=rows))]).astype(np.uint32), ci[keep], v[keep]


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("kind,n", [("units", 64), ("tiles", 8), ("tiles", 136)])
@pytest.mark.parametrize("window", [None, "16", "128", "256"])
def test_lists_in_another_order(kind, n, dt, window, monkeypatch):
    # every tile's columns permuted, its first and last one in place (a list of neighbours still looks like a box), and
    # the tiles of a window in reverse
    if window:
        monkeypatch.setenv("B200SPMM_WINDOW", window)
    rp, ci, v = matrix(kind, dt)
    info, a = arrays(rp, ci, v)
    cw = info.col_window
    lists, tiles = a["tcA2B"].reshape(-1, cw), a["data"].reshape(-1, 16, cw)
    order = np.concatenate([[0], np.arange(cw - 2, 0, -1), [cw - 1]])
    lists, tiles = lists[:, order], tiles[:, :, order]
    for w in range(info.eff_row_windows):
        lo, hi = a["rowOffset"][w], a["rowOffset"][w + 1]
        lists[lo:hi], tiles[lo:hi] = lists[lo:hi][::-1].copy(), tiles[lo:hi][::-1].copy()
    a["tcA2B"], a["data"] = np.ascontiguousarray(lists).ravel(), np.ascontiguousarray(tiles).ravel()
    check(info, a, rp, ci, v, n, True)


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("kind,n", [("units", 64), ("tiles", 8), ("tiles", 136)])
@pytest.mark.parametrize("window", [None, "16", "128", "256"])
def test_values_outside_the_matrix(kind, n, dt, window, monkeypatch):
    # the matrix is said to end five rows and 150 columns (a tile's worth and more, not on a tile's edge) before its
    # stored values do; and the padded slots hold values
    if window:
        monkeypatch.setenv("B200SPMM_WINDOW", window)
    rp, ci, v = matrix(kind, dt)
    info, a = arrays(rp, ci, v)
    cw = info.col_window
    tiles = a["data"].reshape(-1, 16, cw)
    tiles[np.repeat((a["tcA2B"] == PAD).reshape(-1, 1, cw), 16, 1)] = 7
    check(info, a, rp, ci, v, n, False)  # values under padding alone: nothing else is odd about the arrays
    info.rows, info.cols = ROWS - 5, COLS - 150
    check(info, a, *inside(rp, ci, v, ROWS - 5, COLS - 150), n, True)


def test_windows_off_the_grid():
    # one window of rows 5 .. 20 and one of rows 21 .. 36
    rng = np.random.default_rng(1)
    A = np.zeros((40, 64), np.float16)
    A[5:37] = rng.uniform(0.1, 1, (32, 64))
    info, _ = arrays(*matrix("units", np.float16))
    info.rows, info.cols, info.nnzs = 40, 64, 32 * 64
    info.total_row_windows, info.eff_row_windows, info.total_tiles = 3, 2, 8
    a = {"rowOffset": np.array([0, 4, 8], np.uint32), "rowIdx": np.array([5, 21], np.uint32),
         "tcA2B": np.tile(np.arange(64, dtype=np.uint32), 2),
         "data": np.ascontiguousarray(A[5:37].reshape(2, 16, 4, 16).transpose(0, 2, 1, 3)).ravel()}
    rp = np.concatenate([[0], np.cumsum((A != 0).sum(1))]).astype(np.uint32)
    check(info, a, rp, np.nonzero(A)[1].astype(np.uint32), A[A != 0], 64, True)


@pytest.mark.parametrize("what", ["falls", "empty window", "starts late", "another number of tiles", "row past the end", "windows overlap",
                                  "windows swapped", "more windows than tiles"])
def test_bad_tables_are_refused(what):
    info, a = arrays(*matrix("units", np.float16))
    if what == "falls":
        a["rowOffset"][3] = a["rowOffset"][5] + 1
    elif what == "empty window":
        a["rowOffset"][3] = a["rowOffset"][2]
    elif what == "starts late":
        a["rowOffset"][0] = 1
    elif what == "another number of tiles":
        info.total_tiles -= 1
    elif what == "row past the end":
        info.rows = int(a["rowIdx"][-1])
    elif what == "windows overlap":
        a["rowIdx"][1] = a["rowIdx"][0] + 8
    elif what == "windows swapped":
        a["rowIdx"][[1, 2]] = a["rowIdx"][[2, 1]]
    else:
        info.eff_row_windows = info.total_tiles + 1
    with pytest.raises(capi.SpmmError) as e:
        make_plan(info, a)
    assert e.value.status == capi.ERR_INVALID_ARG


@pytest.mark.parametrize("kind", ["units", "tiles"])
@pytest.mark.parametrize("window", [None, "rows", "16"])
def test_windows_of_a_matrix_without_rows_are_refused(kind, window, monkeypatch):
    # by the look over the tables alone: nothing is summed up over rows that are not there
    if window:
        monkeypatch.setenv("B200SPMM_WINDOW", window)
    info, a = arrays(*matrix(kind, np.float16))
    for rows in (0, 16):  # none, and as many as the first window has
        info.rows = rows
        with pytest.raises(capi.SpmmError) as e:
            make_plan(info, a)
        assert e.value.status == capi.ERR_INVALID_ARG


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("shift", [8, 12, 15])
def test_windows_across_the_chunks_of_the_row_sums(dt, shift):
    # windows off the grid of 16 rows: some have rows on both sides of a multiple of 1,024, and far apart windows share a warp
    rng, rows, cols = np.random.default_rng(shift), 6000, 900
    lengths = rng.integers(0, 5, rows)
    lengths[1500:4600] = 0
    lengths[[1007, 1012, 1016]] = [300, 65, 900]
    ci = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in lengths]).astype(np.uint32)
    rp, v = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32), rng.uniform(0.1, 1, ci.size).astype(dt)
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v))
    info = capi.BtcfInfo()
    for k in ("cols", "nnzs", "total_row_windows", "eff_row_windows", "total_tiles", "row_window", "col_window"):
        setattr(info, k, getattr(f, k))
    info.rows = rows + shift
    info.dtype, info.elt_size = (capi.F16, 2) if dt == np.float16 else (capi.TF32, 4)
    a = {k: np.array(getattr(f, k)) for k in ("rowOffset", "tcA2B", "data", "rowIdx")}
    a["rowIdx"] = a["rowIdx"] + np.uint32(shift)
    check(info, a, np.concatenate([np.zeros(shift, np.uint32), rp]), ci, v, 40, True)
