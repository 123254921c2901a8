"""Products in CUDA graphs: a replay runs at the addresses its launches were captured with, whatever the plan did since."""
import numpy as np
import pytest

import hopper_spmm_b200 as hs
from cases import dense_b, random_csr

pytestmark = pytest.mark.gpu

# a matrix, B200SPMM_WINDOW, a width and a wider one: parts of super-windows of 128 and 256 rows, whole ones with B re-laid, windows
# cut between the CTAs of the 16-row kernel, row units with cut rows
SCRATCH = {
    "parts_128": ((1300, 6003, 0.14, 5, np.float16), None, 72, 120),
    "parts_256": ((6000, 3000, 0.15, 5, np.float16), None, 136, 192),
    "re_laid": ((700, 1004, 0.3, 5, np.float32), "128", 128, 328),
    "gathered": ((1300, 6003, 0.14, 5, np.float16), None, 72, 120),  # (B cannot be re-laid)
    "pieces": ((64, 9000, 0.3, 5, np.float32), "16", 64, 192),
    "cut_rows": ((2000, 3000, 0.01, 5, np.float16), "rows", 64, 256),
}


def make(name, monkeypatch):
    (rows, cols, density, seed, dt), window, n, wider = SCRATCH[name]
    if window:
        monkeypatch.setenv("B200SPMM_WINDOW", window)
    m = random_csr(rows, cols, density, seed, dt, dense_rows=[3, rows - 9] if name == "cut_rows" else ())
    if name == "gathered":  # half of the columns are gone
        kept = np.sort(np.random.default_rng(2).permutation(2 * cols)[:cols]).astype(np.uint32)
        cols = 2 * cols
        m = (rows, cols, m[2], kept[m[3]], m[4])
    return hs.CSR2BTCFNOBITMAP(hs.CSR_MTX(*m)), rows, cols, dt, n, wider


@pytest.mark.parametrize("name", list(SCRATCH))
def test_a_graph_outlives_a_wider_product(name, monkeypatch):
    import torch
    f, rows, cols, dt, n, wider = make(name, monkeypatch)
    B = torch.from_numpy(dense_b(cols, wider, 3, dt)).cuda()
    first = B[:, :n].contiguous()
    plan, other = hs.SpmmPlan(f), None
    try:
        want, launches = plan.spmm(first).clone(), plan.launch_info().kernel_launches
        assert launches >= 2  # (the kernel that fills the scratch and the one that reads it)
        g, out = torch.cuda.CUDAGraph(), torch.full((rows, n), float("nan"), device="cuda")
        with torch.cuda.graph(g):
            plan.spmm(first, out, sync=False)
        wide = plan.spmm(B).clone()  # outgrows the scratch of the graph
        other = hs.SpmmPlan(f)       # and somebody else has use for what was freed
        other_wide = other.spmm(B).clone()
        for _ in range(2):
            out.fill_(float("nan"))
            g.replay()
            assert torch.equal(out, want)
            assert torch.equal(plan.spmm(B), wide) and torch.equal(other.spmm(B), other_wide)
        assert torch.equal(wide, other_wide) and torch.equal(plan.spmm(first), want)
    finally:
        plan.close()
        if other is not None:
            other.close()


@pytest.mark.parametrize("name", list(SCRATCH))
def test_a_graph_holds_the_kernels_of_the_call_without_one_before_it(name, monkeypatch):
    # nothing before the capture; then a wider product is the first of its width in a capture
    import torch
    f, rows, cols, dt, n, wider = make(name, monkeypatch)
    B = torch.from_numpy(dense_b(cols, wider, 3, dt)).cuda()
    eager, plan = hs.SpmmPlan(f), hs.SpmmPlan(f)
    try:
        want, ran, graphs = [], [], []
        for w in (n, wider):
            want.append(eager.spmm(B[:, :w].contiguous()).clone())
            ran.append(eager.launch_info())
        for w, info in zip((n, wider), ran):
            b, out = B[:, :w].contiguous(), torch.full((rows, w), float("nan"), device="cuda")
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                plan.spmm(b, out, sync=False)
            got = plan.launch_info()
            assert (got.row_window, got.kernel_launches, got.n_ctas) == (info.row_window, info.kernel_launches, info.n_ctas)
            graphs.append((g, b, out))
        for _ in range(2):
            for (g, _, out), c in zip(graphs, want):
                out.fill_(float("nan"))
                g.replay()
                assert torch.equal(out, c)
        plan.sync()
        assert torch.equal(plan.spmm(B), want[1])
    finally:
        plan.close()
        eager.close()
