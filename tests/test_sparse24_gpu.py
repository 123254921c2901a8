"""256-row super-windows in the tensor core's 2:4 form (fp16): sums that are exact in fp32 have the bits of the dense tiles',
others are no further from 64 bits, and infinities in B stay infinities in the rows that meet them."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
import parity
from cases import random_csr
from hopper_spmm_b200 import synth

pytestmark = pytest.mark.gpu

SPARSE, DENSE = 4, 6  # stages of the ring


def product(monkeypatch, f, B, sparse, n_extra=0, c_half=False):
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "256")
    monkeypatch.setenv("B200SPMM_SPARSE24", "1" if sparse else "0")
    plan = hs.SpmmPlan(f)
    monkeypatch.delenv("B200SPMM_SPARSE24")
    try:
        C = torch.full((f.rows, B.shape[1] + n_extra), float("nan"), device="cuda", dtype=torch.float16 if c_half else torch.float32)
        plan.spmm(B, C[:, : B.shape[1]], c_half=c_half)
        info = plan.launch_info()
        assert info.row_window == 256 and info.stages == (SPARSE if sparse else DENSE)
        assert torch.isnan(C[:, B.shape[1]:]).all()
        return C[:, : B.shape[1]]
    finally:
        plan.close()


def crowded(rows, cols, fill, seed, empty=()):
    """A random matrix with groups of three and four entries, many of them in some rows, and every column in every window."""
    rows, cols, rp, ci, v = random_csr(rows, cols, fill, seed, np.float16, empty_rows=list(empty))
    mask = np.zeros((rows, cols), bool)
    for r in range(rows):
        mask[r, ci[rp[r]:rp[r + 1]]] = True
    full = np.flatnonzero(mask.any(1))
    for lo in range(0, rows, 128):
        live = full[(full >= lo) & (full < lo + 128)]
        if live.size:
            mask[live[np.arange(cols) % live.size], np.arange(cols)] = True
    for r in full[::37]:
        mask[r, 41:48] = True
        mask[r, 200:220:2] = True
        for at in range(516, cols - 20, 1024):
            mask[r, at:at + 8] = True
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.uint32)
    ci = np.nonzero(mask)[1].astype(np.uint32)
    return rows, cols, rp, ci


@pytest.mark.parametrize("rows,cols,fill,n,empty", [(600, 1000, 0.05, 192, [(0, 256)]), (511, 1600, 0.08, 136, []), (256, 1041, 0.04, 256, []),
                                                    (1300, 4080, 0.1, 520, [(512, 768), (1280, 1300)]), (300, 800, 0.03, 264, [])])
def test_exact_sums_have_the_bits_of_the_dense_tiles(rows, cols, fill, n, empty, monkeypatch):
    import torch
    rows, cols, rp, ci = crowded(rows, cols, fill, 7, empty)
    rng = np.random.default_rng(3)
    v = rng.integers(-3, 4, ci.size).astype(np.float16)  # (explicit zeros among them)
    B = torch.from_numpy(rng.integers(-4, 5, (cols, n + 8)).astype(np.float16)).cuda()[:, :n]
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v))
    got, want = product(monkeypatch, f, B, True, 24), product(monkeypatch, f, B, False)
    assert torch.equal(got, want)
    assert torch.equal(product(monkeypatch, f, B, True, c_half=True), want.half())


@pytest.mark.parametrize("fill,cols,n", [(0.07, 3000, 256), (0.1, 4096, 200), (0.12, 2048, 400)])
def test_no_further_from_64_bits_than_dense_tiles(fill, cols, n, monkeypatch):
    import torch
    rows, cols, rp, ci, v = random_csr(700, cols, fill, 5, np.float16)
    v = np.abs(v) + np.float16(0.1)  # of one sign: what the tensor core cuts off adds up
    B = np.abs(np.random.default_rng(2).standard_normal((cols, n))).astype(np.float16)
    dense = np.zeros((rows, cols))
    for r in range(rows):
        dense[r, ci[rp[r]:rp[r + 1]]] = v[rp[r]:rp[r + 1]]
    want = torch.from_numpy(dense).cuda() @ torch.from_numpy(B.astype(np.float64)).cuda()
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v))
    dB = torch.from_numpy(B).cuda()
    off = [float((product(monkeypatch, f, dB, sparse).double() - want).norm() / want.norm()) for sparse in (True, False)]
    assert off[0] <= off[1]
    parity.check(product(monkeypatch, f, dB, True).cpu().numpy(), rows, rp, ci, v, B)


def test_infinities_stay_where_they_are_met(monkeypatch):
    import torch
    rows, cols, rp, ci = crowded(600, 1000, 0.05, 9)
    rng = np.random.default_rng(4)
    v = rng.uniform(0.5, 1, ci.size).astype(np.float16)
    entries = np.zeros((rows, cols), bool)
    for r in range(rows):
        entries[r, ci[rp[r]:rp[r + 1]]] = True
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v))
    n = 136
    B = rng.uniform(0.5, 1, (cols, n)).astype(np.float16)
    at = rng.permutation(cols)[:n]  # one column of the matrix for every feature
    at[:60] = np.arange(40, 100)
    B[at, np.arange(n)] = np.where(np.arange(n) % 2, -np.inf, np.inf)
    got = product(monkeypatch, f, torch.from_numpy(B).cuda(), True).cpu().numpy()
    dense = product(monkeypatch, f, torch.from_numpy(B).cuda(), False).cpu().numpy()
    for k in range(n):
        meet = entries[:, at[k]]
        assert (got[meet, k] == B[at[k], k]).all()
        assert not np.isinf(got[~meet, k]).any()  # finite, or NaN as a dense tile has it
    assert np.isnan(dense[np.isnan(got)]).all()


@pytest.mark.parametrize("rows,cols,fill,width", [(512, 800, 0.1, 200), (300, 6000, 0.02, 40)])
def test_crowded_rows_stay_dense(rows, cols, fill, width, monkeypatch):
    # more of a row in its rest than a block of tiles collects, and than the format has places for
    import torch
    rows, cols, rp, ci = crowded(rows, cols, fill, 3)
    mask = np.zeros((rows, cols), bool)
    for r in range(rows):
        mask[r, ci[rp[r]:rp[r + 1]]] = True
    for at in range(0, cols - width, 600):
        mask[5, at:at + width] = True
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.uint32)
    ci = np.nonzero(mask)[1].astype(np.uint32)
    B = torch.ones((cols, 136), dtype=torch.float16, device="cuda")
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, np.ones(ci.size, np.float16)))
    monkeypatch.setenv("B200SPMM_WINDOW", "256")
    monkeypatch.setenv("B200SPMM_SPARSE24", "1")
    plan = hs.SpmmPlan(f)
    try:
        C = plan.spmm(B)
        assert plan.launch_info().stages == DENSE
        assert torch.equal(C[:, 0].cpu(), torch.from_numpy(mask.sum(1).astype(np.float32)))
    finally:
        plan.close()


def test_large_pruned_matrices_take_it_by_themselves(monkeypatch):
    # the same bits in a graph that is the plan's first launch, and with B fetched through the tensor maps
    import torch
    csr = synth.pruned_weight_csr(16384, 8192, 0.09, seed=3, device="cuda")
    f = hs.DeviceBtcf(csr.rows, csr.cols, csr.row_ptr.to(torch.int32), csr.col_idx, csr.values)
    B = synth.dense_normal(csr.cols, 520, 3, 3, "cuda", torch.float16)
    got = []
    for how in ("graph", "call", "maps"):
        if how == "maps":
            monkeypatch.setenv("B200SPMM_PACK_B", "0")
        plan = hs.SpmmPlan(f)
        try:
            C = torch.full((csr.rows, 520), float("nan"), device="cuda")
            if how == "graph":
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    plan.spmm(B, C, sync=False)
                g.replay()
                torch.cuda.synchronize()
            else:
                plan.spmm(B, C)
            assert plan.launch_info().stages == SPARSE and plan.launch_info().kernel_launches == (1 if how == "maps" else 2)
            got.append(C)
        finally:
            plan.close()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    rp, ci, v = csr.numpy()
    parity.check_rows(torch.cat([got[0][:300], got[0][-300:]]).cpu().numpy(), rp, ci, v, B.cpu().numpy(), [(0, 300), (csr.rows - 300, csr.rows)])


@pytest.mark.parametrize("surplus,at", [(8, 64), (20, 64), (20, 484), (48, 0), (48, 496), (48, 1400)])
def test_what_goes_to_the_rest_may_lie_close_together(surplus, at, monkeypatch):
    # whole groups of four in some rows, two of each in the rest, in one block of 16 tiles (512 columns) or across two; every
    # column in every window, so that groups of the lists are groups of columns
    import torch
    rows, cols, n = 300, 1500, 136
    mask = np.random.default_rng(surplus).random((rows, cols)) < 0.02
    mask[np.arange(cols) % 60, np.arange(cols)] = mask[260 + np.arange(cols) % 40, np.arange(cols)] = True
    for r in (70, 133, 255):
        mask[r] = False
        mask[r, at:at + 2 * surplus] = True
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.uint32)
    ci = np.nonzero(mask)[1].astype(np.uint32)
    rng = np.random.default_rng(3)
    v = rng.choice(np.array([-3, -2, -1, 1, 2, 3], np.float16), ci.size)
    B = torch.from_numpy(rng.integers(-4, 5, (cols, n)).astype(np.float16)).cuda()
    f = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v))
    got = product(monkeypatch, f, B, True)
    assert torch.equal(got, product(monkeypatch, f, B, False))
    dense = np.zeros((rows, cols))
    dense[np.repeat(np.arange(rows), np.diff(rp.astype(np.int64))), ci] = v
    assert torch.equal(got.cpu().double(), torch.from_numpy(dense) @ B.cpu().double())


def test_matrices_beyond_the_limit_do_not_pay_for_the_form(monkeypatch):
    # a twentieth of a row's groups has more than two entries: a sample says so in less than 0.1 ms, the form takes 0.6 ms and more
    import time

    import torch
    csr = synth.pruned_weight_csr(20480, 8192, 0.22, seed=3, device="cuda")
    f = hs.DeviceBtcf(csr.rows, csr.cols, csr.row_ptr.to(torch.int32), csr.col_idx, csr.values)
    B = synth.dense_normal(csr.cols, 256, 3, 3, "cuda", torch.float16)
    took = {}
    for rounds in range(6):
        for env in (None, "0"):
            if env:
                monkeypatch.setenv("B200SPMM_SPARSE24", env)
            else:
                monkeypatch.delenv("B200SPMM_SPARSE24", raising=False)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            plan = hs.SpmmPlan(f)
            torch.cuda.synchronize()
            took.setdefault(env, []).append(time.perf_counter() - t0)
            if not rounds:
                plan.spmm(B)
                assert plan.launch_info().row_window == 256 and plan.launch_info().stages == DENSE
            plan.close()
    assert min(took[None]) - min(took["0"]) < 0.35e-3
    f.close()


def test_weights_that_are_pruned_two_of_four_take_it(monkeypatch):
    # half of all entries, and none in the rest
    import torch
    rows, cols, n = 12288, 8192, 256
    g = torch.Generator(device="cuda").manual_seed(3)
    pairs = torch.tensor([[0, 1], [0, 2], [0, 3], [1, 2], [1, 3], [2, 3]], device="cuda", dtype=torch.int32)
    ci = pairs[torch.randint(0, 6, (rows * cols // 4,), generator=g, device="cuda")] + 4 * (torch.arange(rows * cols // 4, device="cuda", dtype=torch.int32) % (cols // 4))[:, None]
    v = torch.randint(1, 4, (ci.numel(),), generator=g, device="cuda").half()
    f = hs.DeviceBtcf(rows, cols, torch.arange(rows + 1, device="cuda", dtype=torch.int32) * (cols // 2), ci.reshape(-1), v)
    B = torch.randint(-4, 5, (cols, n), generator=g, device="cuda").half()
    plan = hs.SpmmPlan(f)
    try:
        C = plan.spmm(B)
        assert plan.launch_info().row_window == 256 and plan.launch_info().stages == SPARSE
        dense = torch.zeros((rows, cols), device="cuda", dtype=torch.float16)
        dense.scatter_(1, ci.reshape(rows, -1).long(), v.reshape(rows, -1))
        assert torch.equal(C, dense.float() @ B.float())
    finally:
        plan.close()
        f.close()
