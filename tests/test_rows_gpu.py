"""The row-by-row kernel on the device against the CPU oracle, at the sizes where its cuts and lane groups can go
wrong.  B200SPMM_WINDOW=rows sends any matrix down this path; nearly empty tiles take it by themselves."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
import parity
from cases import dense_b

pytestmark = pytest.mark.gpu


def rows_of_lengths(lengths, cols, seed, dt):
    rng = np.random.default_rng(seed)
    ci = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in lengths]).astype(np.uint32)
    v = rng.uniform(-1, 1, ci.size).astype(np.float32).astype(dt)
    v[v == 0] = 1
    return len(lengths), cols, np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32), ci, v


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [8, 24, 40, 64, 104, 128, 136, 520])
def test_batches_units_and_pieces_at_their_edges(dt, n, monkeypatch):
    # whole and ragged batches of four, rows of one unit, rows cut into two, three and many pieces, empty rows at
    # both ends and in between; n covers one lane per row up to a full warp, lanes left over, a narrower last pass
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    lengths = [0, 0, 1, 2, 3, 4, 5, 63, 64, 65, 0, 127, 128, 129, 255, 256, 257, 1000, 0, 7] + [9] * 40 + [0] * 21
    rows, cols, rp, ci, v = rows_of_lengths(lengths, 1013, 3, dt)
    Bfull = torch.from_numpy(dense_b(cols, n + 16, 9, dt)).cuda()
    Bv = Bfull[:, 8:8 + n]
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        Cfull = torch.full((rows, n + 24), float("nan"), device="cuda")  # every row must be written, and nothing else
        plan.spmm(Bv, Cfull[:, 8:8 + n])
        info = plan.launch_info()
        assert info.row_window == 16 and info.stages == 0 and info.kernel_launches == 2
        first = Cfull[:, 8:8 + n].clone()
        parity.check(first.cpu().numpy(), rows, rp, ci, v, Bv.cpu().numpy())
        assert torch.isnan(Cfull[:, :8]).all() and torch.isnan(Cfull[:, 8 + n:]).all()
        plan.spmm(Bv, Cfull[:, 8:8 + n])
        assert torch.equal(first, Cfull[:, 8:8 + n])
        assert torch.equal(plan.spmm(Bv, c_half=True), first.half())
    finally:
        plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [8, 40, 72, 128, 136])
@pytest.mark.parametrize("fill", [0, 0.7, 1.1])
def test_units_walked_by_warps_and_by_groups(dt, n, fill, monkeypatch):
    # long rows of every remainder of a batch and of a warp's groups, among so many short ones that whole warps take all units,
    # the long ones, or none: short rows of up to two batches, `fill` times as many as the GPU's resident warps hold
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    lanes = min(n, 128, 256 // np.dtype(dt).itemsize) * np.dtype(dt).itemsize // 16  # (of a pass: at least two groups a warp)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n_short = int(fill * sms * 32 * (32 // lanes) / -(-n // 128))
    lengths = np.concatenate([[0, 200, 0], np.arange(9, 45), [61, 64, 65, 100, 129, 255, 256, 0], np.arange(n_short) % 8 + 1])
    cols = 1013
    rng = np.random.default_rng(n)
    rp = np.concatenate([[0], np.cumsum(lengths)])
    ci = (np.repeat(rng.integers(0, cols - lengths) - rp[:-1], lengths) + np.arange(rp[-1])).astype(np.uint32)
    v = (rng.choice([-1, 1], ci.size) * rng.uniform(0.1, 1, ci.size)).astype(dt)
    rp = rp.astype(np.uint32)
    B = dense_b(cols, n, 9, dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(lengths.size, cols, rp, ci, v)))
    try:
        dC = torch.full((lengths.size, n), float("nan"), device="cuda")
        plan.spmm(torch.from_numpy(B).cuda(), dC)
        assert plan.launch_info().stages == 0
        parity.check(dC.cpu().numpy(), lengths.size, rp, ci, v, B)
        assert torch.equal(plan.spmm(torch.from_numpy(B).cuda()), dC)
    finally:
        plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_infinities_in_b_reach_the_rows_that_meet_them(dt, monkeypatch):
    # rows with every remainder of a batch, whole and cut (units of 64 entries); every column of B but the last few has
    # an infinity in a row of its own: a row of C is infinite exactly where it has an entry there, and nowhere NaN
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    cols, n = 200, 136
    lengths = list(range(1, 14)) + [61, 62, 63, 64, 65, 66, 67, 129, 130, 131] + [3, 6, 1] * 9
    rows, cols, rp, ci, v = rows_of_lengths(lengths, cols, 8, dt)
    B = dense_b(cols, n, 4, dt)
    hit = np.random.default_rng(5).permutation(cols)[:n - 4]
    B[hit, np.arange(n - 4)] = np.where(np.arange(n - 4) % 2, np.inf, -np.inf).astype(dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        got = plan.spmm(torch.from_numpy(B).cuda()).cpu().numpy()
    finally:
        plan.close()
    bits = (lambda x: x) if dt == np.float16 else (lambda x: (x.view(np.uint32) & np.uint32(0xFFFFE000)).view(np.float32))
    for r in range(rows):
        at = slice(rp[r], rp[r + 1])
        terms = bits(v[at]).astype(np.float64)[:, None] * bits(B[ci[at]]).astype(np.float64)
        want = terms.sum(0)
        assert np.array_equal(got[r][np.isinf(want)], want[np.isinf(want)]), r
        fin = np.isfinite(want)
        assert (np.abs(got[r][fin] - want[fin]) <= len(terms) * 2.0 ** -23 * np.abs(terms).sum(0)[fin]).all(), r  # fp32 sums


@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_a_row_of_one_entry_is_one_exact_product(dt, monkeypatch):
    # its batch is filled up with parts of the value: every finite fp16 value; tf32 values of every exponent, about the
    # powers of two.  Products of 11 bits by 11 are exact in fp32 (those of tf32 that stay normal are compared).
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    if dt == np.float16:
        v = np.arange(1, 65536, dtype=np.uint16).view(np.float16)
    else:
        low = np.array([0, 1, 2, 3, 4, 511, 512, 1022, 1023], np.uint32)
        v = ((np.arange(255, dtype=np.uint32)[:, None] << 10 | low).ravel() << 13).view(np.float32)
        v = np.concatenate([v, -v])
    v = v[np.isfinite(v)]
    rows, cols, n = v.size, 8, 16
    ci = (np.arange(rows) % cols).astype(np.uint32)
    B = dense_b(cols, n, 6, dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, np.arange(rows + 1, dtype=np.uint32), ci, v)))
    try:
        got = plan.spmm(torch.from_numpy(B).cuda()).cpu().numpy()
        assert plan.launch_info().stages == 0
    finally:
        plan.close()
    b = B if dt == np.float16 else (B.view(np.uint32) & np.uint32(0xFFFFE000)).view(np.float32)
    want = v.astype(np.float64)[:, None] * b[ci].astype(np.float64)
    normal = (np.abs(want) >= 2.0 ** -104) & (np.abs(want) < 2.0 ** 127) | (dt == np.float16)  # (the last part's product too)
    assert np.array_equal(got[normal], want[normal])


@pytest.mark.parametrize("dt", [np.float16, np.float32])
def test_bands_and_the_whole_walk_the_same_units(dt, monkeypatch):
    # large enough for bands: the host call goes band by band through a list of its own, the device call through the list
    # of all units; rows without entries in every band, hub rows cut into many pieces, a run of them at one end
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    rng = np.random.default_rng(12)
    lengths = rng.integers(0, 40, 130_007)
    lengths[rng.random(lengths.size) < 0.1] = 0
    lengths[rng.integers(0, lengths.size, 40)] = rng.integers(250, 1100, 40)
    lengths[-5:] = 1001  # (2.5 million entries and rows: bands start at two)
    cols, rp = 1201, np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    start = rng.integers(0, cols - lengths)
    ci = (np.repeat(start - rp[:-1].astype(np.int64), lengths) + np.arange(rp[-1])).astype(np.uint32)  # neighbours: distinct, ascending
    v = rng.uniform(0.1, 1, ci.size).astype(dt)
    B = dense_b(cols, 24, 3, dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(lengths.size, cols, rp, ci, v)))
    try:
        host = plan.spmm_host(B, np.full((lengths.size, 24), np.nan, np.float32))
        assert plan.launch_info().kernel_launches > 2 and plan.launch_info().stages == 0  # bands
        dC = torch.full((lengths.size, 24), float("nan"), device="cuda")
        plan.spmm(torch.from_numpy(B).cuda(), dC)
        assert plan.launch_info().kernel_launches == 2
        assert np.array_equal(host, dC.cpu().numpy())
        parity.check(host, lengths.size, rp, ci, v, B)
    finally:
        plan.close()


@pytest.mark.parametrize("rows,cols", [(1, 5), (17, 1), (3, 4000)])
def test_smallest_matrices(rows, cols, monkeypatch):
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    rows, cols, rp, ci, v = rows_of_lengths([min(cols, 1 + 700 * k) for k in range(rows)], cols, 1, np.float16)
    B = dense_b(cols, 72, 2)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        parity.check(plan.spmm_host(B), rows, rp, ci, v, B)
    finally:
        plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [8, 16, 24, 40, 48])
@pytest.mark.parametrize("rows,cols", [(700, 6001), (149, 2048), (3, 700), (1200, 16500)])
def test_narrow_b_at_the_edges_of_its_column_blocks(dt, n, rows, cols):
    # one column block and several, all in shared memory at once and group by group; CTAs with one row, several rows
    # and none; rows of a few entries, empty ones and rows of many steps
    import torch
    rng = np.random.default_rng(rows + n)
    lengths = rng.integers(cols // 12, cols // 5, rows)
    lengths[[0, rows // 2, rows - 1]] = [0, 5, 33]
    rows, cols, rp, ci, v = rows_of_lengths(lengths, cols, 7, dt)
    Bfull = torch.from_numpy(dense_b(cols, n + 16, 4, dt)).cuda()
    Bv = Bfull[:, 8:8 + n]
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        Cfull = torch.full((rows, n + 8), float("nan"), device="cuda")
        plan.spmm(Bv, Cfull[:, 4:4 + n])
        got = Cfull[:, 4:4 + n].clone()
        assert torch.isnan(Cfull[:, :4]).all() and torch.isnan(Cfull[:, 4 + n:]).all()
        parity.check(got.cpu().numpy(), rows, rp, ci, v, Bv.cpu().numpy())
        assert torch.equal(plan.spmm(Bv, c_half=True), got.half()) and torch.equal(plan.spmm(Bv), got)
    finally:
        plan.close()


@pytest.mark.parametrize("rows,cols,density,n,narrow", [(1290, 777, 0.2, 32, True), (1290, 777, 0.2, 40, False), (2100, 5000, 0.3, 16, True),
                                                        (2100, 5000, 0.3, 24, True), (1300, 8000, 0.14, 32, False)])
def test_narrow_kernel_only_where_it_is_expected_to_be_faster(rows, cols, density, n, narrow):
    # up to three words a row of B always, four where all of B fits
    import torch
    rng = np.random.default_rng(rows)
    rows, cols, rp, ci, v = rows_of_lengths(rng.binomial(cols, density, rows), cols, 7, np.float16)
    B = dense_b(cols, n, 2)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        got = plan.spmm(torch.from_numpy(B).cuda())
        assert (plan.launch_info().threads == 1024) == narrow
        parity.check(got.cpu().numpy(), rows, rp, ci, v, B)
    finally:
        plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [8, 24, 56])
def test_tma_boxes_wider_than_b(dt, n, monkeypatch):
    # the 16-row tile kernel with B narrower than one 128-byte box: the features beyond n arrive as zeros
    monkeypatch.setenv("B200SPMM_WINDOW", "16")
    rows, cols, rp, ci, v = rows_of_lengths([40, 0, 7, 300] * 30 + [1], 500, 5, dt)
    B = dense_b(cols, n, 6, dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        parity.check(plan.spmm_host(B), rows, rp, ci, v, B)
        assert plan.launch_info().tma_gather == 1
    finally:
        plan.close()


@pytest.mark.parametrize("density,rows_kernel", [(0.04, True), (0.07, True), (0.11, False)])
def test_fill_of_the_tiles_decides_between_units_and_tiles(density, rows_kernel):
    # 0.04: 7 % of a tile's slots in use, 0.07: 10 %, and super-windows would wait for too few tiles; 0.11: 13 %
    import torch
    rng = np.random.default_rng(2)
    lengths = rng.binomial(700, density, 600)
    rows, cols, rp, ci, v = rows_of_lengths(lengths, 700, 7, np.float16)
    B = dense_b(cols, 96, 2)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    try:
        got = plan.spmm(torch.from_numpy(B).cuda())
        assert (plan.launch_info().stages == 0) == rows_kernel
        parity.check(got.cpu().numpy(), rows, rp, ci, v, B)
    finally:
        plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("n", [16, 64, 136, 320])
def test_tiles_of_consecutive_columns_read_b_in_boxes(dt, n):
    # dense blocks: B's rows arrive in one box per tile, past its last row in the ragged one; mixed tiles in between
    import torch
    rng = np.random.default_rng(1)
    cols = 1045
    blocks = [np.arange(b, min(b + 29, cols)) for b in (0, 131, 640, cols - 29, cols - 5)]
    per_row = [np.unique(np.concatenate([blocks[(r // 16) % 5], blocks[(r // 48 + 2) % 5], rng.choice(cols, 3)])) for r in range(400)]
    ci = np.concatenate(per_row).astype(np.uint32)
    rp = np.concatenate([[0], np.cumsum([c.size for c in per_row])]).astype(np.uint32)
    v = rng.uniform(0.1, 1, ci.size).astype(np.float32).astype(dt)
    B = dense_b(cols, n, 8, dt)
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(400, cols, rp, ci, v)))
    try:
        dC = torch.full((400, n), float("nan"), device="cuda")
        plan.spmm(torch.from_numpy(B).cuda(), dC)
        assert plan.launch_info().stages > 0
        parity.check(dC.cpu().numpy(), 400, rp, ci, v, B)
    finally:
        plan.close()


def test_the_list_of_the_bands_is_made_for_the_first_host_call():
    # eight bytes a row that a plan of device products does not hold
    import torch
    from hopper_spmm_b200 import _capi as capi
    rows, cols, n = 1 << 23, 1024, 8
    ci = np.random.default_rng(3).integers(0, cols, rows).astype(np.uint32)
    v = np.ones(rows, np.float16)
    B = dense_b(cols, n, 3)
    f = hs.DeviceBtcf(rows, cols, torch.arange(rows + 1, dtype=torch.int32, device="cuda"), torch.from_numpy(ci.view(np.int32)).cuda(), torch.from_numpy(v).cuda())
    plan = hs.SpmmPlan(f)
    try:
        want = plan.spmm(torch.from_numpy(B).cuda(), c_half=True).cpu().numpy()
        assert plan.launch_info().stages == 0 and np.array_equal(want, B[ci])

        def free():
            assert capi.lib().b200spmm_release_cached_memory(0) == 0
            return torch.cuda.mem_get_info()[0]

        before = free()
        assert np.array_equal(plan.spmm_host(B, c_half=True), want)
        assert plan.launch_info().kernel_launches > 2  # bands
        taken = before - free()
        assert taken >= rows * n * 2 + rows * 6  # C, and most of the list
        assert np.array_equal(plan.spmm_host(B, c_half=True), want)
        assert before - free() == taken
    finally:
        plan.close()
        f.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("rows", [1023, 1024, 1025, 3000, 262144, 262145])
def test_running_sums_at_the_edges_of_their_chunks(dt, rows, monkeypatch):
    # chunks of 1,024 rows, as many of them as the one pass takes and one row more; rows of many pieces beside each other, at a
    # chunk's edge and at the end, windows without rows, and a window whose runs are full: the most entries that a warp lists
    import torch
    monkeypatch.setenv("B200SPMM_WINDOW", "rows")
    rng, cols = np.random.default_rng(rows), 5003
    lengths = rng.integers(0, 4, rows)
    lengths[100:180] = 0
    lengths[[5, 6, 511, 1022, rows - 1]] = [5003, 4096, 4097, 65, 2049]
    lengths[192:208] = 700
    ci = np.concatenate([np.arange(k) + 3 if 192 <= r < 208 else np.sort(rng.choice(cols, k, replace=False)) if k > 3 else
                         np.arange(k) * 1000 + r % 1000 for r, k in enumerate(lengths)]).astype(np.uint32)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    v, B = rng.uniform(0.1, 1, ci.size).astype(dt), dense_b(cols, 8, 9, dt)
    dB = torch.from_numpy(B).cuda()
    plan = hs.SpmmPlan(hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    dev = hs.DeviceBtcf(rows, cols, *(torch.from_numpy(a).cuda() for a in (rp.view(np.int32), ci.view(np.int32), v)))
    plan_dev = hs.SpmmPlan(dev)  # its tables are looked over while the units are made
    try:
        C_out = plan.spmm(dB)
        assert plan.launch_info().stages == 0
        parity.check(C_out.cpu().numpy(), rows, rp, ci, v, B)
        assert torch.equal(plan_dev.spmm(dB), C_out)
    finally:
        plan.close()
        plan_dev.close()
        dev.close()
