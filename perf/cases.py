"""The products and conversions that users of this library run, as measurable cases.

A case is a matrix (kind and size), a width of B, an element type, the type C is stored in and the call that
is made (`call`):

* ``device``   a plan is kept, B and C live on the GPU: ``SpmmPlan.spmm``
* ``host``     a plan is kept, B and C are pinned host arrays: ``SpmmPlan.spmm_host``
* ``fresh``    the matrix itself is new at every step (a sampled subgraph, a freshly pruned weight) and lives on
               the GPU as CSR: ``DeviceBtcf``, ``SpmmPlan``, one ``spmm``, and both handles are closed again
* ``load``     CSR in host memory, as read from a checkpoint: ``CSR2BTCFNOBITMAP`` on the host, ``SpmmPlan``, one
               ``spmm`` with B on the GPU

The matrix kinds are those of ``hopper_spmm_b200.synth``: uniform-random sparsity, 16 x 8 blocks, R-MAT graph
adjacency and unstructured pruned weights.
"""
import math

import torch

import hopper_spmm_b200 as hs
from hopper_spmm_b200 import synth


def _case(name, kind, rows, cols, fill, n, dtype="f16", c_half=False, call="device"):
    """`fill`: average degree of a graph, otherwise the share of stored entries."""
    c = {"kind": kind, "rows": rows, "cols": cols, "fill": fill, "n": n, "dtype": dtype, "c_half": c_half, "call": call}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small layer called in a loop: nothing but launch latency
        _case("uniform_1000_n32", "uniform", 1003, 997, 0.02, 32),
        # the first benchmark configuration: one ordinary, still latency-sensitive product
        _case("uniform_4096_n128", "uniform", 4096, 4096, 0.01, 128),
        # the tf32 benchmark configuration: block-sparse matrix, every tile full
        _case("blocks_16384_tf32_n256", "blocks", 16384, 16384, 0.005, 256, dtype="tf32"),
        # one layer of a graph network on a million nodes (benchmark configuration)
        _case("graph_2^20_n64", "graph", 1 << 20, 1 << 20, 16, 64),
        # a full-precision graph model's last layer: node count of no particular form, width of a class count
        _case("graph_150001_tf32_n40", "graph", 150001, 150001, 14, 40, dtype="tf32"),
        # the largest one: 16 M nodes, half a billion entries (the benchmark's default configuration)
        _case("graph_2^24_n128", "graph", 1 << 24, 1 << 24, 32, 128),
        # a pruned linear layer over a long prompt (benchmark configuration)
        _case("pruned_prefill_n2048", "pruned", 28672, 8192, 0.1, 2048),
        # ... over a batch of short ones, activations back in half precision
        _case("pruned_batch_n192", "pruned", 28672, 8192, 0.1, 192, c_half=True),
        # ... and in token-by-token decoding of eight sequences
        _case("pruned_decode_n8", "pruned", 28672, 8192, 0.1, 8, c_half=True),
        # a sampled subgraph per training step: convert, plan, multiply once
        _case("graph_60000_fresh_n128", "graph", 60000, 60000, 12, 128, call="fresh"),
        # the operator as the reference calls it: host arrays in and out, elements in the matrix's type
        _case("graph_2^18_host_n128", "graph", 1 << 18, 1 << 18, 16, 128, c_half=True, call="host"),
        # a pruned weight brought from host memory to its first product when a model is loaded
        _case("pruned_14336_load_n64", "pruned", 14336, 4096, 0.1, 64, call="load"),
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    """A case of the same ranges.  B's width is a multiple of 8 (the library's contract); rows and columns are
    any number."""
    call = rng.choice(["device"] * 7 + ["host", "fresh", "load"])
    kind = rng.choice(["graph", "graph", "pruned", "pruned", "uniform", "blocks"])
    small = call != "device"  # calls that move the matrix or B through the host, or convert, at every pass
    if kind == "graph":
        rows = cols = _log_int(rng, 2000, (1 << 18) if small else (1 << 21))
        fill, n = rng.randint(6, 40), _log_int(rng, 16, 256, 8)
    elif kind == "pruned":
        rows, cols = _log_int(rng, 1024, 14336 if small else 28672), _log_int(rng, 1024, 4096 if small else 8192)
        fill, n = round(rng.uniform(0.05, 0.3), 3), _log_int(rng, 8, 2048, 8)
    elif kind == "uniform":
        rows, cols = _log_int(rng, 256, 8192), _log_int(rng, 256, 8192)
        fill, n = round(math.exp(rng.uniform(math.log(0.003), math.log(0.04))), 4), _log_int(rng, 8, 512, 8)
    else:
        rows, cols = _log_int(rng, 1024, 16384, 16), _log_int(rng, 1024, 16384, 8)
        fill, n = round(math.exp(rng.uniform(math.log(0.002), math.log(0.03))), 4), _log_int(rng, 32, 512, 8)
    dtype = "tf32" if kind == "blocks" and rng.random() < 0.7 or rng.random() < 0.25 else "f16"
    return _case(None, kind, rows, cols, fill, n, dtype, dtype == "f16" and rng.random() < 0.4, call)


def _graph(nodes, degree, seed, dtype):
    """R-MAT adjacency with self-loops (none on the largest graphs) and values 1 / degree(row), for any node
    count: the ids of the next power of two are scaled down to it, which keeps the degree distribution."""
    scale = max(1, (nodes - 1).bit_length())
    keys = synth.rmat_edges(scale, degree * nodes, seed, "cuda")
    if nodes != 1 << scale:
        r, c = (keys >> 32) * nodes >> scale, (keys & 0xFFFFFFFF) * nodes >> scale
        keys = torch.unique((r << 32) | c)
    if nodes <= 1 << 22:
        diag = torch.arange(nodes, dtype=torch.int64, device="cuda")
        keys = torch.unique(torch.cat([keys, (diag << 32) | diag]))
    r = keys >> 32
    row_ptr = torch.zeros(nodes + 1, dtype=torch.int64, device="cuda")
    row_ptr[1:] = torch.cumsum(torch.bincount(r, minlength=nodes), 0)
    inv = (1.0 / (row_ptr[1:] - row_ptr[:-1]).to(torch.float32)).to(dtype)
    return synth.Csr(nodes, nodes, row_ptr, (keys & 0xFFFFFFFF).to(torch.int32), inv[r])


def _matrix(case, seed):
    dtype = torch.float16 if case["dtype"] == "f16" else torch.float32
    rows, cols, fill = case["rows"], case["cols"], case["fill"]
    if case["kind"] == "graph":
        return _graph(rows, fill, seed, dtype)
    make = {"uniform": synth.uniform_random_csr, "blocks": synth.block_clustered_csr, "pruned": synth.pruned_weight_csr}
    m = make[case["kind"]](rows, cols, fill, seed=seed, device="cuda")
    if m.values.dtype != dtype:
        g = torch.Generator(device="cuda").manual_seed(seed)
        new = torch.randn(m.nnz, generator=g, device="cuda") if dtype == torch.float32 else m.values
        m.values = (new * 0.02 if case["kind"] == "pruned" else new).to(dtype)
    return m


def _dense(case, seed):
    make = synth.dense_uniform if case["kind"] in ("graph", "uniform") else synth.dense_normal
    return make(case["cols"], case["n"], seed, 3, "cuda", torch.float16 if case["dtype"] == "f16" else torch.float32)


def prepare(case, seed):
    m = _matrix(case, seed)
    state = {"call": case["call"], "c_half": case["c_half"]}
    csr = (m.rows, m.cols, m.row_ptr.to(torch.int32), m.col_idx, m.values)
    if case["call"] == "load":
        csr = hs.CSR_MTX(m.rows, m.cols, *m.numpy())
    del m
    torch.cuda.empty_cache()  # the library allocates beside torch's pool
    if case["call"] in ("fresh", "load"):
        state["csr"] = csr
    else:
        state["plan"] = hs.SpmmPlan(hs.DeviceBtcf(*csr))
    del csr
    torch.cuda.empty_cache()
    B = _dense(case, seed)
    if case["call"] == "host":
        c_type = torch.float16 if case["c_half"] else torch.float32
        state["pinned"] = (B.cpu().pin_memory(), torch.empty((case["rows"], case["n"]), dtype=c_type).pin_memory())
        state["B"], state["C"] = (t.numpy() for t in state["pinned"])
    else:
        state["B"] = B
    return state


def run(state):
    call, half = state["call"], state["c_half"]
    if call == "device":
        return state["plan"].spmm(state["B"], c_half=half, sync=False)
    if call == "host":
        return state["plan"].spmm_host(state["B"], state["C"], c_half=half)
    fmt = hs.DeviceBtcf(*state["csr"]) if call == "fresh" else hs.CSR2BTCFNOBITMAP(state["csr"])
    plan = hs.SpmmPlan(fmt)
    C = plan.spmm(state["B"], c_half=half)
    plan.close()
    if call == "fresh":
        fmt.close()
    return C


def _entries(case):
    """Stored entries (for graphs: edges drawn, a few per cent of which coincide)."""
    return case["rows"] * case["fill"] if case["kind"] == "graph" else int(case["rows"] * case["cols"] * case["fill"])


def work(case):
    """CSR once (value and 32-bit column per entry, 32-bit row offsets), B once, C once."""
    esz = 2 if case["dtype"] == "f16" else 4
    nnz = _entries(case)
    csr = nnz * (esz + 4) + 4 * (case["rows"] + 1)
    dense = case["cols"] * case["n"] * esz + case["rows"] * case["n"] * (2 if case["c_half"] else 4)
    return {"bytes": csr + dense, "flops": 2 * nnz * case["n"]}


def tolerance(case):
    """fp16 products are exact in fp32 and are summed in fp32 (by tensor cores, whose sums truncate); a result
    stored in half precision carries its rounding.  tf32 keeps ten mantissa bits of both inputs, cut or rounded."""
    if case["dtype"] == "tf32":
        return {"rel": 2e-3}
    return {"rel": 5e-4} if case["c_half"] else {"rel": 5e-5}
