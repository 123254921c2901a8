"""The device-side converter against the host converter (and so the reference algorithm), bit for
bit, and a product computed from a matrix that never left the GPU."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
import parity
from cases import FORMAT_FIELDS, dense_b, random_csr
from hopper_spmm_b200 import _capi as capi
from hopper_spmm_b200 import synth

pytestmark = pytest.mark.gpu


def device_convert(rows, cols, rp, ci, v, rw=16, cw=0):
    import torch
    d = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).view(dt).copy()).cuda()
    vals = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    return hs.DeviceBtcf(rows, cols, d(rp, np.int32), d(ci, np.int32), vals, row_window=rw, col_window=cw)


def assert_same(dev, host):
    got = dev.to_host()
    assert (dev.eff_row_windows, dev.total_tiles) == (host.eff_row_windows, host.total_tiles)
    for k in FORMAT_FIELDS:
        assert np.array_equal(got[k].view(np.uint8), np.ascontiguousarray(getattr(host, k)).view(np.uint8)), k


@pytest.mark.parametrize("dt,cw", [(np.float16, 16), (np.float32, 8), (np.float32, 4)])
@pytest.mark.parametrize("rw", [8, 16])
def test_matches_host_converter(dt, cw, rw):
    shapes = [(1, 1, 1.0), (16, 16, 0.5), (17, 33, 0.2), (203, 517, 0.03), (500, 70000, 0.0005), (96, 7, 0.6)]
    for seed, (rows, cols, dens) in enumerate(shapes):
        rows, cols, rp, ci, v = random_csr(rows, cols, dens, seed, dt, empty_rows=[(16, 48)] if rows > 64 else (),
                                           dense_rows=[3] if cols < 1000 and rows > 3 else ())
        host = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v), row_window=rw, col_window=cw)
        dev = device_convert(rows, cols, rp, ci, v, rw, cw)
        assert_same(dev, host)
        dev.close()


@pytest.mark.parametrize("name,k", [("uniform_4096_fp16", 0), ("blocks_16384_tf32", 1), ("rmat24_sharded_fp16", 6)])
def test_benchmark_matrices(name, k):
    csr, _ = synth.make_config(name, 0, "cpu", k)
    rp, ci, v = csr.numpy()
    host = hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(csr.rows, csr.cols, rp, ci, v))
    dev = device_convert(csr.rows, csr.cols, rp, ci, v)
    assert_same(dev, host)


def test_empty_matrix():
    rp = np.zeros(41, np.uint32)
    dev = device_convert(40, 10, rp, np.zeros(0, np.uint32), np.zeros(0, np.float16))
    assert (dev.eff_row_windows, dev.total_tiles, dev.total_row_windows) == (0, 0, 3)


def test_unsorted_or_repeated_columns_are_refused():
    rp = np.array([0, 3], np.uint32)
    for ci in ([5, 2, 9], [2, 5, 5], [2, 5, 99]):
        with pytest.raises(capi.SpmmError) as e:
            device_convert(1, 16, rp, np.array(ci, np.uint32), np.ones(3, np.float16))
        assert e.value.status == capi.ERR_BAD_CSR


def test_product_from_a_matrix_that_stayed_on_the_gpu():
    import torch
    csr, B = synth.make_config("rmat24_sharded_fp16", 0, "cuda", 8)  # generated on the device
    dev = hs.DeviceBtcf(csr.rows, csr.cols, csr.row_ptr.to(torch.int32), csr.col_idx, csr.values)
    plan = hs.SpmmPlan(dev)
    C_dev = plan.spmm(B)
    rp, ci, v = csr.numpy()
    parity.check(C_dev.cpu().numpy(), csr.rows, rp, ci, v, B.cpu().numpy())
    plan.close()


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("rows,cols,per_row", [(50, 255, 40), (50, 256, 40), (50, 257, 40), (33, 66000, 900), (40, 520001, 3000),
                                               (3001, 300000, 3), (700, 900001, 2000)])
def test_window_by_window_and_through_the_sort(dt, rows, cols, per_row):
    # a bit set of one group, its edges, several groups a thread, a set above 48 KB; windows too empty for a set and
    # rows too long for one.  Rows of very different length, empty ones in between
    rng = np.random.default_rng(cols)
    lengths = np.minimum(rng.integers(0, 2 * per_row + 1, rows), cols)
    lengths[rows // 2] = min(cols, 40 * per_row)
    ci = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in lengths]).astype(np.uint32)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    v = rng.uniform(0.5, 1, ci.size).astype(np.float32).astype(dt)
    dev = device_convert(rows, cols, rp, ci, v)
    assert_same(dev, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    dev.close()
    bad = []
    for at in (rp[rows // 2], rp[rows // 2] + 1):  # a column out of range, two columns out of order
        c = ci.copy()
        c[at] = cols if at == rp[rows // 2] else c[at - 1]
        bad.append((rp, c))
    r = rp.copy()
    r[rows // 2] += 1 + r[rows // 2 + 1] - r[rows // 2]  # row pointers that fall
    bad += [(r, ci), (np.concatenate([rp[:-1], [rp[-1] - 1]]).astype(np.uint32), ci), (np.concatenate([[1], rp[1:]]).astype(np.uint32), ci)]
    for r, c in bad:
        with pytest.raises(capi.SpmmError) as e:
            device_convert(rows, cols, r, c, v)
        assert e.value.status == capi.ERR_BAD_CSR


def test_bit_set_that_just_fits_48_kb():
    # with the kernel's own shared variables it does not: in a process where no larger set has run before
    import subprocess
    import sys
    code = """if True:
        import numpy as np, torch, hopper_spmm_b200 as hs
        cols, ci = 348_519, np.arange(17, 348_519, 500, dtype=np.int32)
        d = lambda a: torch.from_numpy(a).cuda()
        dev = hs.DeviceBtcf(1, cols, d(np.array([0, ci.size], np.int32)), d(ci), d(np.ones(ci.size, np.float16)))
        got = dev.to_host()["tcA2B"]
        assert np.array_equal(got[:ci.size], ci.view(np.uint32)) and (got[ci.size:] == 0xFFFFFFFF).all()
    """
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)


@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("rows,cols,nnz", [(100, 300, 1023), (100, 300, 1024), (100, 300, 1025), (65536, 64, 20000), (65552, 64, 20000),
                                           (262144, 300, 300000), (262145, 300, 300000), (40000, 3000, 1100000), (40000, 3000, 2200000)])
def test_entries_at_the_edges_of_the_window_passes(dt, rows, cols, nnz):
    # entries a block places at a time; windows a round of the scan takes, the most that one block scans; a tile array made ahead
    # and one that would be larger than that (tf32 from 1.04e6 entries on, fp16 from 2.08e6)
    rng = np.random.default_rng(nnz + rows)
    flat = np.sort(rng.choice(rows * cols, nnz, replace=False))
    rp = np.searchsorted(flat, np.arange(rows + 1, dtype=np.int64) * cols).astype(np.uint32)
    ci, v = (flat % cols).astype(np.uint32), rng.uniform(0.1, 1, nnz).astype(dt)
    dev = device_convert(rows, cols, rp, ci, v)
    assert_same(dev, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    dev.close()


@pytest.mark.parametrize("dt,rw,cw", [(np.float16, 16, 0), (np.float32, 16, 0), (np.float16, 8, 4)])
def test_windows_at_the_edges_of_the_sorts_and_the_set(dt, rw, cw):
    # entries of a window that a warp sorts with two, four and eight keys a lane, and that a block marks; among the last both lists
    counts = [0, 1, 2, 63, 64, 65, 127, 128, 129, 0, 255, 256, 257, 4095, 4096, 4097, 9001, 1, 300, 64]
    rng, cols = np.random.default_rng(7), 3001
    lengths, ci = [], []
    for n in counts:
        cuts = np.sort(rng.integers(0, n + 1, rw - 1)) if n < 4000 else np.arange(1, rw) * n // rw  # (rows of up to `cols` entries)
        lengths += list(np.diff(np.concatenate([[0], cuts, [n]])))
    ci = np.concatenate([np.sort(rng.choice(cols if k % 3 else min(cols, 2 * n + 1), n, replace=False)) for k, n in enumerate(lengths)]).astype(np.uint32)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    v, rows = rng.uniform(0.1, 1, ci.size).astype(dt), len(lengths)
    dev = device_convert(rows, cols, rp, ci, v, rw, cw)
    assert_same(dev, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v), row_window=rw, **({"col_window": cw} if cw else {})))
    dev.close()
    for n in (2, 65, 129, 300, 4096):  # a column out of order, one twice, one out of range
        for c in ([3, 1], [5, 5], [7, cols]):
            bad, at = ci.copy(), int(rp[counts.index(n) * rw] if n != 300 else rp[18 * rw])
            r = int(np.searchsorted(rp, at, side="right")) - 1
            while lengths[r] < 2:
                r += 1
            bad[rp[r]:rp[r] + 2] = c
            with pytest.raises(capi.SpmmError) as e:
                device_convert(rows, cols, rp, bad, v, rw, cw)
            assert e.value.status == capi.ERR_BAD_CSR


@pytest.mark.parametrize("rw", [8, 16])
@pytest.mark.parametrize("cols", [3001, 743000])
def test_windows_of_up_to_512_entries_and_every_width_of_the_set(rw, cols):
    # of 743,000 columns, where a block has one set, warps sort them with sixteen keys a lane; else blocks mark them
    counts = [257, 511, 512, 513, 300, 0, 384, 512, 256, 4097]
    rng, lengths, ci = np.random.default_rng(rw), [], []
    for n in counts:
        cuts = np.sort(rng.integers(0, n + 1, rw - 1)) if n < 4000 else np.arange(1, rw) * n // rw
        lengths += list(np.diff(np.concatenate([[0], cuts, [n]])))
    for k, n in enumerate(lengths):
        row = np.sort(rng.choice(cols if k % 3 else min(cols, 2 * n + 1), n, replace=False))
        if n > 1:
            row[0], row[-1] = 0, cols - 1
        ci.append(row)
    ci = np.concatenate(ci).astype(np.uint32)
    rp, v, rows = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32), rng.uniform(0.1, 1, ci.size).astype(np.float16), len(lengths)
    dev = device_convert(rows, cols, rp, ci, v, rw)
    assert_same(dev, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v), row_window=rw))
    dev.close()
    for w in (1, 2):  # a column out of order, one twice, one out of range
        for c in ([3, 1], [5, 5], [7, cols]):
            bad, r = ci.copy(), w * rw
            while lengths[r] < 2:
                r += 1
            bad[rp[r]:rp[r] + 2] = c
            with pytest.raises(capi.SpmmError) as e:
                device_convert(rows, cols, rp, bad, v, rw)
            assert e.value.status == capi.ERR_BAD_CSR


def test_tiles_made_ahead_are_no_more_than_every_column_in_every_window():
    # 1.9e6 entries, whose tiles could take 61 MB if they shared no column, and take 12
    import torch
    rng = np.random.default_rng(5)
    rows = cols = 2400
    mask = rng.random((rows, cols)) < 0.34
    rp = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.uint32)
    ci = np.nonzero(mask)[1].astype(np.uint32)
    v = rng.uniform(0.1, 1, ci.size).astype(np.float16)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (rp, ci, v)]

    def free():
        torch.cuda.synchronize()
        assert capi.lib().b200spmm_release_cached_memory(0) == 0
        return torch.cuda.mem_get_info()[0]

    hs.DeviceBtcf(rows, cols, *dev).close()
    before = free()
    f = hs.DeviceBtcf(rows, cols, *dev)
    assert_same(f, hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(rows, cols, rp, ci, v)))
    needed = f.total_tiles * (512 + 64)
    assert before - free() <= needed + (34 << 20)  # (the pool takes 32 MB and more at a time; the tables)
    f.close()
    assert before - free() == 0
