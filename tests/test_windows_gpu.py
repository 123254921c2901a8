"""The kernel of single warps (16-row windows) on the device: against the CPU oracle, and bit for bit against the
pipelined 16-row kernel, which adds the products of a window in the same order and cuts them the same way.  Matrices of
short windows take it by themselves; B200SPMM_WINDOW=warps asks for it."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
import parity
from cases import dense_b, random_csr
from hopper_spmm_b200 import synth

pytestmark = pytest.mark.gpu


def plans(monkeypatch, f):
    """One for this kernel, one for the pipelined kernel with whole windows (a single CTA cuts none)."""
    monkeypatch.setenv("B200SPMM_WINDOW", "warps")
    mine = hs.SpmmPlan(f)
    monkeypatch.setenv("B200SPMM_WINDOW", "16")
    return mine, hs.SpmmPlan(f, n_ctas=1)


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [8, 24, 32, 40, 64, 72, 96, 136, 264])
def test_every_width_of_b(dt, n, monkeypatch):
    # windows of none to 40 tiles (stages of one, two and four, the last one partly filled), ragged last tiles, rows and
    # columns of no multiple of the tile's, windows missing at both ends and between
    import torch
    rows, cols, rp, ci, v = random_csr(715, 317, 0.03, 11, dt, empty_rows=[(0, 35), (256, 384), (700, 715)], dense_rows=[140, 141, 500])
    B = torch.from_numpy(dense_b(cols, n, 3, dt)).cuda()
    mine, other = plans(monkeypatch, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        for half in (False, True):
            got, want = (torch.full((rows, n), float("nan"), device="cuda", dtype=torch.float16 if half else torch.float32) for _ in range(2))
            mine.spmm(B, got, c_half=half)
            info = mine.launch_info()
            assert (info.threads, info.row_window, info.kernel_launches) == (128, 16, 1)
            other.spmm(B, want, c_half=half)
            assert torch.equal(got, want)  # every row written
        parity.check(mine.spmm(B).cpu().numpy(), rows, rp, ci, v, B.cpu().numpy())
    finally:
        mine.close()
        other.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("rows,cols", [(1, 1), (16, 16), (17, 15), (33, 1000)])
def test_single_windows_and_strided_operands(dt, rows, cols, monkeypatch):
    import torch
    rows, cols, rp, ci, v = random_csr(rows, cols, 1.0, 4, dt)
    Bfull = torch.from_numpy(dense_b(cols, 56, 3, dt)).cuda()
    Cfull = torch.full((rows, 72), float("nan"), device="cuda")
    Bv, Cv = Bfull[:, 8:48], Cfull[:, 16:56]
    mine, other = plans(monkeypatch, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        mine.spmm(Bv, Cv)
        assert mine.launch_info().threads == 128
        assert torch.equal(Cv, other.spmm(Bv))
        assert torch.isnan(Cfull[:, :16]).all() and torch.isnan(Cfull[:, 56:]).all()
    finally:
        mine.close()
        other.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_a_callers_arrays_and_infinities(dt, monkeypatch):
    # tiles in the caller's order (the plan keeps an image of its own); padded slots read no row of B
    import torch
    rows, cols, rp, ci, v = random_csr(80, 50, 0.3, 6, dt)
    m = hs.DeviceBtcf(rows, cols, torch.from_numpy(rp.view(np.int32)).cuda(), torch.from_numpy(ci.view(np.int32)).cuda(), torch.from_numpy(v).cuda())
    B = dense_b(cols, 40, 3, dt)
    unused = np.setdiff1d(np.arange(cols), ci[rp[0]:rp[16]])
    B[unused[:1]] = np.inf  # no entry of the first window meets it, if there is such a column
    mine, other = plans(monkeypatch, m)
    try:
        dB = torch.from_numpy(B).cuda()
        got, want = mine.spmm(dB), other.spmm(dB)
        assert mine.launch_info().threads == 128
        assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want)) and torch.equal(got.isnan(), want.isnan())
        assert torch.isfinite(got[:16]).all()
    finally:
        mine.close()
        other.close()


def test_matrices_of_short_windows_choose_it_by_themselves():
    import torch
    for cols, n in ((4096, 128), (16384, 64)):
        m = synth.block_clustered_csr(1024, cols, 0.005, seed=3, device="cuda")
        f = hs.DeviceBtcf(m.rows, m.cols, m.row_ptr.to(torch.int32), m.col_idx, m.values)
        plan = hs.SpmmPlan(f)
        try:
            B = synth.dense_normal(cols, n, 3, 3, "cuda", m.values.dtype)
            C = plan.spmm(B)
            assert plan.launch_info().threads == 128
            rp, ci, v = m.numpy()
            parity.check(C.cpu().numpy(), m.rows, rp, ci, v, B.cpu().numpy())
        finally:
            plan.close()


@pytest.mark.parametrize("dt,n", [(np.float16, 256), (np.float32, 128)])
@pytest.mark.parametrize("lead,tail", [(1, 1), (1024, 0), (2, 1024)])
def test_long_gaps_are_not_cleared_by_warps_of_two_lines(dt, n, lead, tail, monkeypatch):
    # a warp clears what is missing behind its window (and ahead of the first one), twice as slowly where it has two lines
    import torch
    m = synth.block_clustered_csr(16384, 8192, 0.005, seed=3, device="cuda")
    ptr = m.row_ptr.to(torch.int32)
    ptr = torch.cat([torch.zeros(16 * lead, dtype=torch.int32, device="cuda"), ptr, ptr[-1:].expand(16 * tail)])
    rows, v = 16384 + 16 * (lead + tail), m.values.to(torch.float16 if dt == np.float16 else torch.float32)
    f = hs.DeviceBtcf(rows, m.cols, ptr, m.col_idx, v)
    B = synth.dense_normal(m.cols, n, 3, 3, "cuda", v.dtype)
    plan = hs.SpmmPlan(f)
    monkeypatch.setenv("B200SPMM_WINDOW", "16")
    other = hs.SpmmPlan(f, n_ctas=1)
    try:
        got, want = (torch.full((rows, n), float("nan"), device="cuda") for _ in range(2))
        plan.spmm(B, got)
        info = plan.launch_info()
        line = 64 if dt == np.float16 else 32
        if lead + tail < 8:
            assert (info.threads, info.feature_slab) == (128, 2 * line)
        else:
            assert info.threads != 128 or info.feature_slab == line
        other.spmm(B, want)
        assert torch.equal(got, want)
    finally:
        plan.close()
        other.close()
