"""Performance cases: what a program that uses this library has it do, through its public entry points.

Four paths:
  spmm     C = A·B with a packed matrix and a plan that the program keeps (``engine.spmm``), every
           encoding, plain and compensated products, with and without the ReLU epilogue
  pack     a device CSR matrix to one of the packed encodings plus the execution plan for it
           (``engine.pack_*`` and ``.plan()``), with or without a row reorder: what every new graph,
           every sampled subgraph and every re-weighted matrix costs
  train    the sparse products of one step of a two-layer graph network through the caller-level
           backend (``mask_b200.spmm_backend``): forward with A, backward with A^T, at the hidden
           width and at the number of classes (often odd)
  session  C = A·B with B and C in pinned host memory (the host-buffer session of the C ABI)

Matrices: ``uniform`` (random positions), ``rmat`` (power-law graph with self-loops, symmetric for
``spmm``, ``pack`` and ``session``, directed for ``train``), ``mesh`` (27-point stencil on a cube;
``shuffled``: its nodes numbered at random, as meshes come from generators and files).  They are
drawn on the GPU from the seed alone.
"""
import ctypes
import math

import torch

from mask_b200 import _lib, engine, spmm_backend

DEVICE = "cuda"


def listed():
    return [
        # the smallest product of the benchmark: a 4096-node matrix, where launches and host time count
        dict(name="uniform-4k", path="spmm", graph="uniform", rows=4096, cols=4096, degree=21.0, N=512, format="srbcrs", tf32x3=False, relu=False),
        # finite-element matrix: dense tiles, neighbouring windows share the rows of B
        dict(name="mesh-100", path="spmm", graph="mesh", rows=1000000, cols=1000000, degree=27.0, N=512, format="srbcrs", tf32x3=False, relu=False),
        # hidden layer of a graph network on a graph of a million nodes
        dict(name="graph-1M", path="spmm", graph="rmat", rows=1 << 20, cols=1 << 20, degree=16.0, N=512, format="srbcrs", tf32x3=False, relu=True),
        # the largest product of the benchmark's sweep
        dict(name="graph-4M", path="spmm", graph="rmat", rows=1 << 22, cols=1 << 22, degree=32.0, N=512, format="srbcrs", tf32x3=False, relu=False),
        # the narrow end of the same sweep
        dict(name="graph-2M-narrow", path="spmm", graph="rmat", rows=1 << 21, cols=1 << 21, degree=20.0, N=64, format="srbcrs", tf32x3=False, relu=False),
        # the COO encoding at a usual feature width, a graph of odd size
        dict(name="graph-300k-metcf", path="spmm", graph="rmat", rows=300007, cols=300007, degree=14.0, N=128, format="metcf", tf32x3=False, relu=False),
        # the bitmap encoding, rectangular and ragged: a panel of rows of a sampled bipartite graph
        dict(name="uniform-100k-mco", path="spmm", graph="uniform", rows=100003, cols=70001, degree=10.0, N=100, format="mco", tf32x3=False, relu=False),
        # FP32-level accuracy asked for
        dict(name="graph-200k-tf32x3", path="spmm", graph="rmat", rows=200000, cols=200000, degree=16.0, N=256, format="srbcrs", tf32x3=True, relu=False),
        # a new graph of a million nodes: format builder and plan
        dict(name="pack-1M", path="pack", graph="rmat", rows=1 << 20, cols=1 << 20, degree=16.0, format="srbcrs", reorder="none"),
        # a mesh with its nodes in no useful order: reverse Cuthill-McKee, then pack and plan
        dict(name="pack-rcm-mesh", path="pack", graph="shuffled", rows=64000, cols=64000, degree=27.0, format="srbcrs", reorder="row_rcm"),
        # the sparse half of a training step, 128 hidden features and 47 classes
        dict(name="train-130k", path="train", graph="rmat", rows=130000, cols=130000, degree=15.0, N=128, classes=47, format="srbcrs"),
        # operands in host memory
        dict(name="session-200k", path="session", graph="rmat", rows=200000, cols=200000, degree=16.0, N=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _matrix(rng, most_rows, most_nnz, graphs, square):
    graph = rng.choice(graphs)
    if graph in ("mesh", "shuffled"):
        g = int(round(_log(rng, 256, min(most_rows, most_nnz / 27.0)) ** (1.0 / 3.0)))
        return dict(graph=graph, rows=g ** 3, cols=g ** 3, degree=27.0)
    rows = int(_log(rng, 256, most_rows))
    degree = round(min(_log(rng, 3.0, 40.0), most_nnz / rows, rows / 8.0), 2)
    cols = rows if (square or graph == "rmat" or rng.random() < 0.5) else int(rows * _log(rng, 0.25, 4.0))
    return dict(graph=graph, rows=rows, cols=cols, degree=max(degree, 1.0))


def draw(rng):
    path = rng.choice(["spmm"] * 5 + ["pack"] * 2 + ["train"] * 2 + ["session"])
    if path == "spmm":
        fmt = rng.choice(["srbcrs", "srbcrs", "metcf", "mco"])
        N = 4 * int(round(_log(rng, 8, 512) / 4))
        c = _matrix(rng, min(1 << 21, (1 << 30) // N), 3.2e7, ["uniform", "rmat", "rmat", "mesh"], False)
        return dict(path=path, **c, N=N, format=fmt, tf32x3=fmt == "srbcrs" and rng.random() < 0.25, relu=rng.random() < 0.3)
    if path == "pack":
        reorder = rng.choice(["none", "none", "row_rcm", "first_col_sort", "jaccard_greedy"])
        fmt = "srbcrs" if reorder != "none" else rng.choice(["srbcrs", "metcf", "mco"])
        graphs = ["shuffled", "rmat"] if reorder == "row_rcm" else ["uniform", "rmat", "mesh", "shuffled"]
        c = _matrix(rng, 1 << 17 if reorder == "row_rcm" else 1 << 20, 2e6 if reorder != "none" else 1.7e7, graphs, reorder == "row_rcm")
        return dict(path=path, **c, format=fmt, reorder=reorder)
    if path == "train":
        c = _matrix(rng, 1 << 18, 4e6, ["uniform", "rmat", "rmat"], True)
        return dict(path=path, **c, N=int(_log(rng, 16, 300)), classes=int(_log(rng, 2, 150)), format=rng.choice(["srbcrs", "srbcrs", "metcf"]))
    N = 4 * int(round(_log(rng, 16, 512) / 4))
    c = _matrix(rng, min(1 << 19, (1 << 26) // N), 4e6, ["uniform", "rmat"], False)
    return dict(path=path, **c, N=N)


# ---- inputs ------------------------------------------------------------------------------------
def _keys_uniform(gen, M, K, nnz):
    return torch.randint(0, M * K, (nnz,), generator=gen, device=DEVICE, dtype=torch.int64)


def _keys_rmat(gen, n, nnz, symmetric):
    """R-MAT (a, b, c, d) = (.57, .19, .19, .05) on the next power of two, scaled to n nodes, plus self-loops."""
    samples = nnz // 2 if symmetric else nnz
    bits = max(1, (n - 1).bit_length())
    src = torch.zeros(samples, dtype=torch.int64, device=DEVICE)
    dst = torch.zeros(samples, dtype=torch.int64, device=DEVICE)
    for _ in range(bits):
        r = torch.rand(samples, generator=gen, device=DEVICE)
        src.mul_(2).add_(r >= 0.76)
        dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    if n != 1 << bits:
        src, dst = (src * n) >> bits, (dst * n) >> bits
    loops = torch.arange(n, dtype=torch.int64, device=DEVICE) * (n + 1)
    return torch.cat([src * n + dst, dst * n + src, loops] if symmetric else [src * n + dst, loops])


def _keys_mesh(gen, n, shuffled):
    g = int(round(n ** (1.0 / 3.0)))
    i = torch.arange(n, dtype=torch.int64, device=DEVICE)
    z, y, x = i // (g * g), (i // g) % g, i % g
    name = torch.randperm(n, generator=gen, device=DEVICE) if shuffled else i
    keys = []
    for d in range(27):
        zz, yy, xx = z + d // 9 - 1, y + (d // 3) % 3 - 1, x + d % 3 - 1
        ok = (zz >= 0) & (zz < g) & (yy >= 0) & (yy < g) & (xx >= 0) & (xx < g)
        keys.append((name * n + name[(zz * g * g + yy * g + xx).clamp_(0, n - 1)])[ok])
    return torch.cat(keys)


def _csr(keys, M, K):
    """Sorted, deduplicated keys row * K + col -> rowptr, colind (int32)."""
    keys = torch.unique(keys)
    rows = keys // K
    colind = (keys - rows * K).to(torch.int32)
    rowptr = torch.zeros(M + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(torch.bincount(rows, minlength=M), 0, out=rowptr[1:])
    return rows, rowptr.to(torch.int32), colind


def _graph(case, gen, symmetric=True, pattern=None, turn=0):
    """CSR on the GPU.  ``pattern``: a generator of its own for the positions; ``turn``: the whole
    16-row windows are moved round by that many."""
    M, K = case["rows"], case["cols"]
    values_gen, gen = gen, pattern or gen
    nnz = int(M * case["degree"])
    if case["graph"] == "uniform":
        keys = _keys_uniform(gen, M, K, nnz)
    elif case["graph"] == "rmat":
        keys = _keys_rmat(gen, M, nnz, symmetric)
    else:
        keys = _keys_mesh(gen, M, case["graph"] == "shuffled")
    gen = values_gen
    if turn:
        whole = M // 16 * 16
        rows = keys // K
        keys += torch.where(rows < whole, (rows + 16 * turn) % max(whole, 1) - rows, 0) * K
    rows, rowptr, colind = _csr(keys, M, K)
    if case["graph"] == "rmat":     # normalised adjacency, as graph networks use it, times a random edge weight
        deg = (rowptr[1:] - rowptr[:-1]).float()
        values = torch.rsqrt(deg[rows].clamp_(min=1) * deg[colind.long()].clamp_(min=1))
        values *= torch.rand(values.shape, generator=gen, device=DEVICE) + 0.5
    elif case["graph"] == "uniform":
        values = torch.rand(colind.shape, generator=gen, device=DEVICE) * 2 - 1
    else:                           # stencil coefficients: off-diagonals U(0.5, 1.5), diagonal 27
        values = torch.rand(colind.shape, generator=gen, device=DEVICE) + 0.5
        values[rows == colind] = 27.0
    return rowptr, colind, values


def _transpose(rowptr, colind, values, M):
    rows = torch.repeat_interleave(torch.arange(M, device=DEVICE), (rowptr[1:] - rowptr[:-1]).long())
    order = torch.argsort(colind.long() * M + rows)
    counts = torch.bincount(colind, minlength=M)
    rp = torch.zeros(M + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(counts, 0, out=rp[1:])
    return rp.to(torch.int32), rows[order].to(torch.int32), values[order]


def _normal(gen, *shape):
    return torch.randn(shape, generator=gen, device=DEVICE)


class _Session:
    """The C ABI's host-buffer session, as a host program holds it."""

    def __init__(self, M, K, rowptr, colind, values):
        self.lib, self.handle = _lib.lib(), ctypes.c_void_p()
        rp, ci, va = rowptr.cpu(), colind.cpu(), values.cpu()
        _lib.check(self.lib.mask_session_create_csr(M, K, ci.numel(), rp.data_ptr(), ci.data_ptr(), va.data_ptr(),
                                                    _lib.POLICY["auto"], ctypes.byref(self.handle)), "mask_session_create_csr")

    def spmm(self, B, C):
        _lib.check(self.lib.mask_session_spmm_host(self.handle, B.data_ptr(), C.data_ptr(), B.shape[1], None), "mask_session_spmm_host")
        return C

    def __del__(self):
        if self.handle:
            self.lib.mask_session_destroy(self.handle)
            self.handle = None


_PACK = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}
_BACKEND = {"srbcrs": spmm_backend.srbcrs_spmm, "metcf": spmm_backend.dtc_spmm}


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    M, K, path = case["rows"], case["cols"], case["path"]
    if path == "pack":
        # another seed gives other values and, without a reorder, other windows in other places, but as
        # many tiles, so that the packed arrays of two seeds are of one size
        pattern = torch.Generator(device=DEVICE)
        pattern.manual_seed(M + K)
        turn = seed % 1009 + 1 if case["reorder"] == "none" else 0
        return dict(case=case, csr=_graph(case, gen, pattern=pattern, turn=turn))
    rowptr, colind, values = _graph(case, gen, symmetric=path != "train")
    N = case["N"]
    if path == "spmm":
        packed = _PACK[case["format"]](rowptr, colind, values, M, K)
        return dict(case=case, packed=packed, plan=packed.plan(), B=_normal(gen, K, N))
    if path == "session":
        B = torch.empty((K, N), pin_memory=True).copy_(_normal(gen, K, N))
        C = torch.empty((M, N), pin_memory=True)
        return dict(case=case, session=_Session(M, K, rowptr, colind, values), B=B, C=C)
    # train: the graph and its transpose have met the backend before (it packs a graph on first sight)
    fwd, bwd = (rowptr, colind, values), _transpose(rowptr, colind, values, M)
    state = dict(case=case, fwd=fwd, bwd=bwd, x1=_normal(gen, M, N), x2=_normal(gen, M, case["classes"]),
                 g2=_normal(gen, M, case["classes"]), g1=_normal(gen, M, N))
    for csr in (fwd, bwd):
        _BACKEND[case["format"]](*csr, state["x2"], M, case["classes"], M)
    return state


def run(state):
    case, path = state["case"], state["case"]["path"]
    if path == "spmm":
        return engine.spmm(state["packed"], state["B"], relu=case["relu"], tf32x3=case["tf32x3"])
    if path == "session":
        return state["session"].spmm(state["B"], state["C"])
    M = case["rows"]
    if path == "train":
        spmm = _BACKEND[case["format"]]
        return [spmm(*state[csr], state[x], M, state[x].shape[1], M)
                for csr, x in (("fwd", "x1"), ("fwd", "x2"), ("bwd", "g2"), ("bwd", "g1"))]
    more = {"reorder": case["reorder"]} if case["reorder"] != "none" else {}
    packed = _PACK[case["format"]](*state["csr"], M, case["cols"], **more)
    packed.plan()
    names = {"srbcrs": ("val_soff", "val_sidx", "val_block_val"),
             "metcf": ("val_soff", "val_sidx", "val_coo_off", "val_coo_idx", "val_coo_val"),
             "mco": ("val_soff", "val_sidx", "val_mco_off", "val_mco_mask", "val_mco_val")}[case["format"]]
    out = {n: getattr(packed, n) for n in names}
    if packed.row_order is not None:
        out["row_order"] = packed.row_order
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------
def _nnz(case):
    M, K, degree = case["rows"], case["cols"], case["degree"]
    if case["graph"] == "uniform":
        return M * K * -math.expm1(M * degree * math.log1p(-1.0 / (M * K)))
    if case["graph"] == "rmat":     # about a tenth of the samples fall on one another
        return 0.9 * M * degree + M
    g = round(M ** (1.0 / 3.0))
    return float((3 * g - 2) ** 3)


def work(case):
    """The matrix as CSR (8 bytes an entry) and each row of B that it touches once, C once; a pack reads
    the CSR and writes what any encoding of it has to hold (a column and a value per entry)."""
    M, K, nnz = case["rows"], case["cols"], _nnz(case)
    csr = 8.0 * nnz + 4.0 * (M + 1)
    if case["path"] == "pack":
        return {"bytes": 2 * csr + (8.0 * M if case["reorder"] != "none" else 0.0), "flops": 0.0}
    touched = K * -math.expm1(-nnz / K) if case["graph"] == "uniform" else K
    widths = [case["N"]] if case["path"] != "train" else [case["N"], case["classes"]] * 2
    return {"bytes": sum(csr + 4.0 * n * (touched + M) for n in widths), "flops": sum(2.0 * nnz * n for n in widths)}


def tolerance(case):
    """Packed arrays are whole numbers and copied values.  Products multiply in TF32 (10-bit mantissas,
    rounded or cut off) with 32-bit sums, or with compensated products at 32-bit accuracy."""
    if case["path"] == "pack":
        return "exact"
    return {"rel": 1e-5} if case.get("tf32x3") else {"rel": 1e-3}
