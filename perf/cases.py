"""Performance cases of graphalgo_gb300: what a program that uses the package has it do.

Every case goes through the public Python entry points, on graphs of the kinds
the package is used on: R-MAT graphs (power-law degrees), Erdos-Renyi graphs
and symmetrised k-nearest-neighbour graphs, with any number of vertices.
Handles and the context are made once (`prepare`) and kept, as a program
keeps them; `run` is one call and returns its results whole. Results on the
device go to buffers that the program keeps, sized for the largest result, with
the number of entries in use beside them.

Kinds of case:
  tc      triangle count, total and per row
  ktruss  one k-truss
  sweep   every k-truss from k = 3 on, each from the one before
  mxm     one masked product C<M> = A*B
  level   one breadth-first level in operator form: the next frontier by the
          complemented product, and the visited set that takes it in
  bc      betweenness centrality of a batch of sources
  batch   triangle counts and 4-trusses of many graphs in one union
  build   edge list on the host to a device CSR, then the lower triangle and
          the symmetric matrix from it
"""
import math

import numpy as np
import torch

import graphalgo_gb300 as ga

_DTYPES = {"int32": (torch.int32, ga.INT32), "int64": (torch.int64, ga.INT64), "fp32": (torch.float32, ga.FP32),
           "fp64": (torch.float64, ga.FP64), "uint8": (torch.uint8, ga.UINT8)}
_TYPESTR = {ga.INT32: "<i4", ga.INT64: "<i8", ga.FP32: "<f4", ga.FP64: "<f8", ga.UINT8: "|u1"}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call there is: a 1,000-vertex graph, where launches and
        # host round trips count
        {"name": "tc_er1000", "kind": "tc", "graph": "er", "n": 1000, "degree": 10, "algo": "msa", "dtype": "uint8"},
        # triangle count of a large power-law graph
        {"name": "tc_rmat18", "kind": "tc", "graph": "rmat", "n": 1 << 18, "degree": 16, "algo": "tri",
         "dtype": "int32"},
        # a k-truss request on a small resident graph
        {"name": "ktruss_rmat12", "kind": "ktruss", "graph": "rmat", "n": 1 << 12, "degree": 16, "algo": "tri",
         "k": 5},
        # a k-truss of a large graph
        {"name": "ktruss_rmat18", "kind": "ktruss", "graph": "rmat", "n": 1 << 18, "degree": 16, "algo": "tri",
         "k": 4},
        # the whole truss decomposition of a large graph, the benchmark's workload
        {"name": "sweep_rmat18", "kind": "sweep", "graph": "rmat", "n": 1 << 18, "degree": 16, "algo": "tri"},
        # the k-truss support product by the reference's default variant
        {"name": "support_msa_rmat18", "kind": "mxm", "shape": "support", "graph": "rmat", "n": 1 << 18,
         "degree": 16, "algo": "msa"},
        # a weighted directed product in double precision, odd and rectangular sizes
        {"name": "mxm_mca_fp64", "kind": "mxm", "shape": "general", "rows": 50021, "inner": 65537, "cols": 40009,
         "degree": 12, "mask_degree": 24, "algo": "mca", "dtype": "fp64"},
        # one level of a 64-source search written with the operators
        {"name": "level_rmat16", "kind": "level", "graph": "rmat", "n": 1 << 16, "degree": 16, "sources": 64,
         "visited": 0.3, "frontier": 0.05},
        # a served betweenness request: 32 sources on a small nearest-neighbour graph
        {"name": "bc32_knn10000", "kind": "bc", "graph": "knn", "n": 10000, "degree": 30, "dim": 14, "sources": 32},
        # betweenness of 64 sources on a large graph
        {"name": "bc64_rmat20", "kind": "bc", "graph": "rmat", "n": 1 << 20, "degree": 16, "sources": 64},
        # many small graphs of uneven size in one call
        {"name": "batch512_knn", "kind": "batch", "count": 512, "least": 32, "most": 4096, "degree": 30, "k": 4},
        # graph preparation from an edge list in host memory
        {"name": "build_rmat18", "kind": "build", "n": 1 << 18, "degree": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tc", "ktruss", "sweep", "mxm", "level", "bc", "batch", "build"])
    if kind in ("tc", "ktruss", "bc"):
        # a k-truss of an Erdos-Renyi graph of these degrees is empty
        graph = rng.choice(["rmat", "rmat", "knn"] if kind == "ktruss" else ["rmat", "rmat", "er", "knn"])
        most = {"rmat": 1 << 18, "er": 200000, "knn": 20000}[graph]
        least, thin = (1000, 8) if kind == "ktruss" else (200, 4)
        case = {"kind": kind, "graph": graph, "n": _log_int(rng, least, most), "degree": rng.randint(thin, 16)}
        if graph == "knn":
            case["degree"], case["dim"] = 30, rng.randint(4, 16)
        if kind == "tc":
            case["algo"] = rng.choice(["msa", "dot", "tri", "tri"])
            case["dtype"] = rng.choice(["int32", "uint8"])
        elif kind == "ktruss":
            case["algo"] = rng.choice(["tri", "tri", "tri", "msa", "hybrid"])
            case["k"] = rng.randint(3, 8)
        else:
            case["sources"] = min(_log_int(rng, 1, 256), case["n"] // 4)
        return case
    if kind == "sweep":
        return {"kind": "sweep", "graph": "rmat", "n": _log_int(rng, 500, 200000), "degree": rng.randint(4, 16),
                "algo": "tri"}
    if kind == "mxm":
        algo = rng.choice(["msa", "msa", "mca", "heap", "dot", "hybrid"])
        if rng.random() < 0.4:
            return {"kind": "mxm", "shape": "support", "graph": rng.choice(["rmat", "er"]),
                    "n": _log_int(rng, 500, 100000), "degree": rng.randint(4, 16), "algo": algo}
        return {"kind": "mxm", "shape": "general", "rows": _log_int(rng, 100, 60000),
                "inner": _log_int(rng, 100, 60000), "cols": _log_int(rng, 100, 60000), "degree": rng.randint(2, 16),
                "mask_degree": rng.randint(2, 32), "algo": algo, "dtype": rng.choice(sorted(_DTYPES))}
    if kind == "level":
        return {"kind": "level", "graph": "rmat", "n": _log_int(rng, 500, 1 << 16), "degree": rng.randint(4, 16),
                "sources": _log_int(rng, 1, 200), "visited": rng.uniform(0.05, 0.6),
                "frontier": rng.uniform(0.001, 0.05)}
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 8, 512), "least": 32, "most": _log_int(rng, 200, 4096),
                "degree": rng.randint(8, 30), "k": rng.randint(3, 8)}
    return {"kind": "build", "n": _log_int(rng, 500, 1 << 18), "degree": rng.randint(4, 16)}


# ------------------------------------------------------------------ the inputs
_state = {}


def _context():
    """The program's one context, on a stream of its own, and that stream."""
    if not _state:
        stream = torch.cuda.Stream()
        _state["stream"] = stream
        _state["ctx"] = ga.Context(0, stream=stream.cuda_stream)
    return _state["ctx"], _state["stream"]


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _pairs(rows, cols, count, g):
    """`count` R-MAT index pairs (0.57, 0.19, 0.19, 0.05), those inside rows x cols."""
    levels = max(1, (max(rows, cols) - 1).bit_length())
    r = torch.zeros(count, dtype=torch.int64, device="cuda")
    c = torch.zeros(count, dtype=torch.int64, device="cuda")
    for _ in range(levels):
        x = torch.rand(count, generator=g, device="cuda")
        r = r * 2 + (x >= 0.76)
        c = c * 2 + (((x >= 0.57) & (x < 0.76)) | (x >= 0.95))
    # a shorter side takes the leading bits
    r >>= levels - max(1, (rows - 1).bit_length())
    c >>= levels - max(1, (cols - 1).bit_length())
    inside = (r < rows) & (c < cols)
    return r[inside], c[inside]


def _edges(case, g):
    """Undirected edges (u, v) of the case's graph; loops and repeats may occur."""
    n, degree = case["n"], case["degree"]
    if case["graph"] == "rmat":
        return _pairs(n, n, n * degree, g)
    if case["graph"] == "er":
        want = min(n * degree, n * (n - 1) // 4)
        u = torch.randint(n, (2 * want + 64,), generator=g, device="cuda")
        v = torch.randint(n, (2 * want + 64,), generator=g, device="cuda")
        key = torch.unique((torch.maximum(u, v) * n + torch.minimum(u, v))[u != v])
        key = key[torch.randperm(len(key), generator=g, device="cuda")[:want]]
        return key // n, key % n
    points = torch.randn(n, case["dim"], generator=g, device="cuda")
    k = min(degree, n - 1)
    near = [torch.cdist(p, points).topk(k + 1, largest=False).indices for p in points.split(4096)]
    near = torch.cat(near)
    return torch.arange(n, device="cuda").repeat_interleave(k + 1), near.reshape(-1)


def _csr_of_keys(key, rows, cols):
    """(rows, cols, rst, col) of sorted distinct keys row * cols + col."""
    row = torch.div(key, cols, rounding_mode="floor")
    rst = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    rst[1:] = torch.cumsum(torch.bincount(row, minlength=rows), 0)
    return rows, cols, rst, key - row * cols


def _symmetric(case, seed):
    """The case's graph as a symmetric CSR without loops or repeats."""
    u, v = _edges(case, _generator(seed, 1))
    n = case["n"]
    u, v = u[u != v], v[u != v]
    return _csr_of_keys(torch.unique(torch.cat([u * n + v, v * n + u])), n, n)


def _values(dtype, count, g):
    t = _DTYPES[dtype][0]
    if t.is_floating_point:
        return 1 - torch.rand(count, generator=g, device="cuda", dtype=torch.float64).to(t)  # edge weights in (0, 1]
    return torch.randint(1, 10, (count,), generator=g, device="cuda").to(t)


def _upload(ctx, m, n, rst, col, val=None, dtype=ga.INT32):
    return ga.Csr.upload(ctx, m, n, rst.to(torch.int32).cpu().numpy(), col.to(torch.int32).cpu().numpy(),
                         None if val is None else val.cpu().numpy(), dtype)


def _general(case, seed):
    """A (rows x inner), B (inner x cols), M (rows x cols): CSRs, and the values of A and B."""
    out = []
    sizes = [("rows", "inner", "degree"), ("inner", "cols", "degree"), ("rows", "cols", "mask_degree")]
    for salt, (r, c, d) in enumerate(sizes):
        rows, cols = case[r], case[c]
        g = _generator(seed, 10 + salt)
        i, j = _pairs(rows, cols, rows * case[d], g)
        csr = _csr_of_keys(torch.unique(i * cols + j), rows, cols)
        out.append(csr + ((_values(case["dtype"], len(csr[3]), g),) if salt < 2 else ()))
    return out


def _level(case, seed):
    """A graph, the frontier with its path counts and the visited set with its."""
    graph = _symmetric(case, seed)
    n, ns = case["n"], case["sources"]
    g = _generator(seed, 20)
    seen = torch.unique(torch.randint(n * ns, (max(1, int(case["visited"] * n * ns)),), generator=g, device="cuda"))
    count = torch.randint(1, 50, (len(seen),), generator=g, device="cuda").to(torch.float64)
    share = min(1.0, case["frontier"] / case["visited"])
    front = torch.rand(len(seen), generator=g, device="cuda") < share
    return graph, _csr_of_keys(seen[front], n, ns) + (count[front],), _csr_of_keys(seen, n, ns) + (count,)


def _sources(case, seed):
    return torch.randperm(case["n"], generator=_generator(seed, 2), device="cuda")[:case["sources"]].cpu().numpy()


def prepare(case, seed):
    ctx, stream = _context()
    kind = case["kind"]
    state = {"case": case, "ctx": ctx, "stream": stream, "out": _buffers(case)}
    if kind in ("tc", "ktruss", "sweep", "bc") or (kind == "mxm" and case["shape"] == "support"):
        state["A"] = _upload(ctx, *_symmetric(case, seed), dtype=_DTYPES[case.get("dtype", "int32")][1])
        if kind == "bc":
            state["sources"] = _sources(case, seed)
    elif kind == "mxm":
        A, B, M = _general(case, seed)
        dtype = _DTYPES[case["dtype"]][1]
        state["A"], state["B"] = _upload(ctx, *A, dtype=dtype), _upload(ctx, *B, dtype=dtype)
        state["M"] = _upload(ctx, *M)
    elif kind == "level":
        graph, front, seen = _level(case, seed)
        state["A"] = _upload(ctx, *graph, dtype=ga.FP64)
        state["F"], state["V"] = _upload(ctx, *front, dtype=ga.FP64), _upload(ctx, *seen, dtype=ga.FP64)
    elif kind == "batch":
        r = np.random.default_rng(seed)
        sizes = r.integers(case["least"], case["most"] + 1, case["count"])
        state["U"], state["voff"] = ga.gen_knn_batch(ctx, sizes, r.integers(4, 17, case["count"]), case["degree"],
                                                     seed)
    else:
        u, v = _pairs(case["n"], case["n"], case["n"] * case["degree"], _generator(seed, 1))
        state["src"], state["dst"] = u.to(torch.int32).cpu().numpy(), v.to(torch.int32).cpu().numpy()
    return state


def _most(case):
    """Stored entries that the case's symmetric graph can have."""
    n, degree = case["n"], case["degree"]
    return min(2 * n * (degree + (case.get("graph") == "knn")), n * n)


_STAGES = 256  # trusses of a sweep that the result buffers hold


def _room(case):
    """Row starts, entries and value type (None: the pattern alone) of every matrix that the case's call returns."""
    kind = case["kind"]
    if kind == "ktruss" or (kind == "mxm" and case["shape"] == "support"):
        return [(case["n"] + 1, _most(case), "int32")]
    if kind == "sweep":
        # the trusses together hold up to about 2.5 log2(n) times the graph's entries
        return [(_STAGES * (case["n"] + 1), int(4 * math.log2(case["n"])) * _most(case), None)]
    if kind == "mxm":
        return [(case["rows"] + 1, case["rows"] * case["mask_degree"], case["dtype"])]
    if kind == "level":
        return [(case["n"] + 1, case["n"] * case["sources"], "fp64")] * 2
    if kind == "batch":
        n = case["count"] * case["most"]
        return [(n + 1, 2 * case["degree"] * n, "int32")]
    if kind == "build":
        return [(case["n"] + 1, _most(case), "int32")] * 3
    return []


def _buffers(case):
    return [[torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.zeros(entries, dtype=torch.int32, device="cuda")] +
            ([torch.zeros(entries, dtype=_DTYPES[dtype][0], device="cuda")] if dtype else [])
            for rows, entries, dtype in _room(case)]


# ------------------------------------------------------------------ one pass
class _View:
    """Device memory of a handle for torch; keeps the handle."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


def _keep(C, out, at=(0, 0)):
    """Copies a device CSR (as many of its arrays as there are buffers) into `out` from `at` on; the place after it."""
    m, _, nnz, dtype = C.info()
    ends = (at[0] + m + 1, at[1] + nnz)
    for ptr, count, typestr, buf, begin in zip(C.device_ptrs(), (m + 1, nnz, nnz), ("<i4", "<i4", _TYPESTR[dtype]), out,
                                               (at[0], at[1], at[1])):
        count = min(count, len(buf) - begin)
        if count > 0:
            buf[begin:begin + count].copy_(torch.as_tensor(_View(C, ptr, count, typestr), device="cuda"))
    return ends


def run(state):
    case, ctx, out = state["case"], state["ctx"], state["out"]
    kind = case["kind"]
    if kind == "tc":
        total, rows = ga.tc(case["algo"], state["A"])
        return [total, rows]
    if kind == "bc":
        return [ga.bc(state["A"], state["sources"])]
    with torch.cuda.stream(state["stream"]):
        if kind == "ktruss":
            C, iterations = ga.ktruss(case["algo"], state["A"], case["k"])
            return [iterations, _keep(C, out[0])[1]] + out
        if kind == "sweep":  # every truss's edges (their values are ones)
            steps, at = np.zeros((_STAGES, 3), np.int64), (0, 0)
            for i, (k, C, iterations) in enumerate(ga.ktruss_sweep(case["algo"], state["A"], 3)):
                at = _keep(C, out[0], at)
                steps[min(i, _STAGES - 1)] = k, iterations, at[1]
            return [steps] + out
        if kind == "mxm":
            A = state["A"]
            C = ga.mxm_masked(case["algo"], A, state.get("B", A), state.get("M", A))
            return [_keep(C, out[0])[1]] + out
        if kind == "level":
            N = ga.mxm_cmask(state["A"], state["F"], state["V"])
            S = ga.add_nointersect(state["V"], N)
            return [_keep(N, out[0])[1], _keep(S, out[1])[1]] + out
        if kind == "batch":
            counts = ga.batch_tc("msa", state["U"], state["voff"])
            K, iterations = ga.batch_ktruss("tri", state["U"], state["voff"], case["k"])
            return [counts, iterations, _keep(K, out[0])[1]] + out
        n = case["n"]
        A = ga.csr_from_edges(ctx, n, n, state["src"], state["dst"],
                              flags=ga.EDGES_MIRROR | ga.EDGES_DROP_LOOPS | ga.EDGES_UNIT)
        L = ga.extract_lower(A)
        S = ga.symm_from_lower(L)
        return [_keep(A, out[0])[1], _keep(L, out[1])[1], _keep(S, out[2])[1]] + out


# ------------------------------------------------------------------ the work
def _entries(case):
    """Stored entries of the case's symmetric graph, about."""
    n, degree = case["n"], case["degree"]
    if case["graph"] == "knn":
        return 1.46 * min(degree, n - 1) * n
    return min((1.82 if case["graph"] == "rmat" else 2.0) * n * degree, n * (n - 1))


def _products(case):
    """Gustavson products of the graph's square, about."""
    z, n = _entries(case), case["n"]
    if case["graph"] != "rmat":
        return z * z / n
    return 0.5 * (2.0 * n * case["degree"]) ** 2 * 0.635 ** math.log2(n)


def work(case):
    kind = case["kind"]
    if kind in ("tc", "ktruss", "sweep"):
        z, n = _entries(case), case["n"]
        if kind == "tc":
            return {"bytes": 4 * (n + z) + 8 * n, "flops": 0}
        if kind == "ktruss":
            return {"bytes": 8 * z + 4 * n + 8 * z * 0.8 + 4 * n, "flops": 0}
        # the trusses together hold about twice log2(n) times the graph's entries
        return {"bytes": 8 * z + 4 * n + 2 * math.log2(n) * (8 * z + 4 * n), "flops": 0}
    if kind == "mxm":
        if case["shape"] == "support":
            z, n = _entries(case), case["n"]
            return {"bytes": 16 * z + 8 * n, "flops": 2 * _products(case)}
        size = {"int32": 4, "int64": 8, "fp32": 4, "fp64": 8, "uint8": 1}[case["dtype"]]
        za, zb, zm = (case[r] * case[d] for r, d in (("rows", "degree"), ("inner", "degree"),
                                                     ("rows", "mask_degree")))
        return {"bytes": (za + zb) * (4 + size) + zm * (8 + size) + 4 * (case["inner"] + 3 * case["rows"]),
                "flops": 2.0 * za * zb / case["inner"]}
    if kind == "level":
        z, n = _entries(case), case["n"]
        pairs = n * case["sources"]
        front, seen = case["frontier"] * pairs, case["visited"] * pairs
        found = min(pairs - seen, front * z / n)
        return {"bytes": 12 * (z + front + 2 * seen + 2 * found) + 20 * n, "flops": 2 * front * z / n}
    if kind == "bc":
        z, n, ns = _entries(case), case["n"], case["sources"]
        return {"bytes": 4 * (z + n) + 8 * n + 4 * ns, "flops": 4.0 * z * ns}
    if kind == "batch":
        n = case["count"] * (case["least"] + case["most"]) / 2
        z = 1.46 * case["degree"] * n
        return {"bytes": 8 * z + 4 * n + 16 * case["count"] + 8 * z * 0.9 + 4 * n, "flops": 0}
    z = 1.82 * case["n"] * case["degree"]
    return {"bytes": 8 * case["n"] * case["degree"] + 8 * (2.5 * z) + 12 * case["n"], "flops": 0}


# ------------------------------------------------------------------ in 64 bits
def _rows_of(rst):
    return torch.repeat_interleave(torch.arange(len(rst) - 1, device="cuda"), rst[1:] - rst[:-1])


def _expand(A, B, most=1 << 25):
    """The products of A * B in pieces: (key row * cols + col, value)."""
    arst, acol, aval = A[2], A[3], A[4].to(torch.float64)
    brst, bcol, bval, cols = B[2], B[3], B[4].to(torch.float64), B[1]
    arow = _rows_of(arst)
    count = brst[acol + 1] - brst[acol]
    ends = torch.cumsum(count, 0)
    total = int(ends[-1]) if len(ends) else 0
    cuts = torch.searchsorted(ends, torch.arange(most, total, most, device="cuda")) if total > most else ends[:0]
    cuts = [0] + cuts.tolist() + [len(acol)]
    for a, b in zip(cuts, cuts[1:]):
        if a >= b:
            continue
        c = count[a:b]
        which = torch.repeat_interleave(torch.arange(a, b, device="cuda"), c)
        first = (torch.cumsum(c, 0) - c).repeat_interleave(c)
        j = brst[acol[which]] + torch.arange(len(which), device="cuda") - first
        yield arow[which] * cols + bcol[j], aval[which] * bval[j]


def _masked_sums(A, B, mask, others=None):
    """Sums of the products at the sorted keys `mask`; the other products go to the list `others`."""
    sums = torch.zeros(len(mask), dtype=torch.float64, device="cuda")
    for key, v in _expand(A, B):
        at = torch.searchsorted(mask, key).clamp(max=len(mask) - 1)
        hit = mask[at] == key
        sums.index_add_(0, at[hit], v[hit])
        if others is not None:
            others.append((key[~hit], v[~hit]))
    return sums


def _padded(x, count):
    return torch.cat([x, x.new_zeros(count - len(x))])


def exact(case, seed):
    kind = case["kind"]
    if kind == "mxm" and case["shape"] == "general" and _DTYPES[case["dtype"]][0].is_floating_point:
        A, B, M = _general(case, seed)
        return [None, [None, None, _padded(_masked_sums(A, B, _rows_of(M[2]) * M[1] + M[3]), _room(case)[0][1])]]
    if kind == "level":
        graph, F, V = _level(case, seed)
        A = graph + (torch.ones(len(graph[3]), dtype=torch.float64, device="cuda"),)
        seen = _rows_of(V[2]) * V[1] + V[3]
        others = [(seen[:0], V[4][:0])]
        _masked_sums(A, F, seen, others)
        key, val = (torch.cat(x) for x in zip(*others))
        found, where = torch.unique(key, return_inverse=True)
        sums = torch.zeros(len(found), dtype=torch.float64, device="cuda").index_add_(0, where, val)
        order = torch.argsort(torch.cat([seen, found]))
        both = torch.cat([V[4], sums])[order]
        return [None, None] + [[None, None, _padded(x, r[1])] for x, r in zip((sums, both), _room(case))]
    if kind == "bc":
        n, _, rst, col = _symmetric(case, seed)
        src = torch.from_numpy(_sources(case, seed)).cuda()
        ns = len(src)
        A = torch.sparse_csr_tensor(rst, col, torch.ones(len(col), dtype=torch.float64, device="cuda"), (n, n))
        sigma = torch.zeros(n, ns, dtype=torch.float64, device="cuda")
        level = torch.full((n, ns), -1, dtype=torch.int32, device="cuda")
        at = torch.arange(ns, device="cuda")
        sigma[src, at], level[src, at] = 1.0, 0
        front, depth = sigma.clone(), 0
        while True:
            front = A @ front
            front[level >= 0] = 0
            reached = front > 0
            if not bool(reached.any()):
                break
            depth += 1
            level[reached] = depth
            sigma += front
        del front
        delta = torch.zeros_like(sigma)
        for d in range(depth, 1, -1):  # a source's own score takes nothing from its searches
            w = A @ torch.where(level == d, (1 + delta) / sigma, 0.0)
            delta += torch.where(level == d - 1, w * sigma, 0.0)
        return [delta.sum(1)]
    return None
