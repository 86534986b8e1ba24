"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the package's public entry points: the reference-shaped
one-shot call on host arrays, solves on a graph that stays on the device (pull in
the exact-order and in the blocked form, push), the call that allocates nothing,
batched personalized PageRank, the uneven multi-graph batch, CSR SpMV and the
multicolour Gauss-Seidel smoother.  Graphs are RMAT, Erdos-Renyi or Chung-Lu
graphs made on the GPU from the seed with plain torch; matrices are 27-point
stencils with varying coefficients, or graphs with random values.
"""
import math

import numpy as np
import torch

import gardenia_ocl_b200 as G

DEV = "cuda"
DAMP = float(np.float32(0.85))
RMAT = (0.57, 0.19, 0.19)
# share of RMAT edge draws that are left after self-loops and repeats are dropped
KEPT = 0.95
# edges from which the blocked layout is the one to build (include/gpr.h, GPR_FORM_AUTO)
BLOCKED_EDGES = 3 << 24


def listed():
    return [
        # The reference driver's own shape: PageRank(m, nnz, ...) once, on host arrays,
        # RMAT with 65,536 vertices, edge factor 16, tolerance 1e-4.
        {"name": "call_host_64k", "kind": "call", "m": 65536, "ef": 16, "tol": 1e-4},
        # A small graph solved again and again with the reference's defaults
        # (EPSILON 1e-3, MAX_ITER 30): launches and barriers count.
        {"name": "pull_10k", "kind": "pull", "m": 10007, "ef": 16, "tol": 1e-3},
        # An ordinary graph on the device, solved to 1e-6.
        {"name": "pull_1m", "kind": "pull", "m": 1000003, "ef": 16, "tol": 1e-6},
        # RMAT with 2^24 vertices, edge factor 16, in the blocked form that the tuner picks.
        {"name": "pull_16m", "kind": "pull", "m": 1 << 24, "ef": 16, "tol": 1e-6},
        # The push direction.
        {"name": "push_3m", "kind": "push", "m": 3000017, "ef": 16, "tol": 1e-6},
        # A caller whose allocator owns the device: CSR on the device, no allocation.
        {"name": "noalloc_250k", "kind": "noalloc", "m": 250007, "ef": 16, "tol": 1e-4},
        # Personalized PageRank: few seeds on a large graph, many on a smaller one.
        {"name": "ppr_4m_k8", "kind": "ppr", "m": 1 << 22, "ef": 16, "k": 8, "tol": 1e-6},
        {"name": "ppr_1m_k100", "kind": "ppr", "m": 1000003, "ef": 16, "k": 100, "tol": 1e-6},
        # 512 graphs of 1,000 to 500,000 vertices, half Erdos-Renyi and half Chung-Lu.
        {"name": "batch_512", "kind": "batch", "graphs": 512, "m_min": 1000, "m_max": 500000,
         "tol": 1e-6},
        # y = A x with the 27-point stencil on 128^3, and with a graph's adjacency.
        {"name": "spmv_stencil_128", "kind": "spmv_stencil", "nx": 128, "ny": 128, "nz": 128},
        {"name": "spmv_graph_2m", "kind": "spmv_graph", "m": 2500009, "ef": 16},
        # Two smoother sweeps, as a multigrid cycle does before it restricts.
        {"name": "symgs_128", "kind": "symgs", "nx": 128, "ny": 128, "nz": 128, "sweeps": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "pull", "pull", "pull", "push", "noalloc", "ppr", "ppr", "batch",
                       "spmv_stencil", "spmv_graph", "symgs"])
    ef = rng.randint(8, 24)
    tol = rng.choice([1e-3, 1e-4, 1e-5, 1e-6])
    if kind == "call":
        return {"kind": kind, "m": _log(rng, 10000, 500000), "ef": ef, "tol": tol}
    if kind == "pull":
        return {"kind": kind, "m": _log(rng, 5000, 10000000), "ef": ef, "tol": tol}
    if kind == "push":
        return {"kind": kind, "m": _log(rng, 100000, 4000000), "ef": ef, "tol": tol}
    if kind == "noalloc":
        return {"kind": kind, "m": _log(rng, 10000, 1000000), "ef": ef, "tol": tol}
    if kind == "ppr":
        return {"kind": kind, "m": _log(rng, 100000, 3000000), "ef": ef,
                "k": _log(rng, 2, 128), "tol": tol}
    if kind == "batch":
        return {"kind": kind, "graphs": _log(rng, 16, 512), "m_min": 1000,
                "m_max": _log(rng, 10000, 300000), "tol": tol}
    if kind == "spmv_graph":
        return {"kind": kind, "m": _log(rng, 50000, 4000000), "ef": ef}
    top = 160 if kind == "spmv_stencil" else 128
    case = {"kind": kind}
    for d in ("nx", "ny", "nz"):
        case[d] = _log(rng, 24, top)
    if kind == "symgs":
        case["sweeps"] = rng.randint(1, 3)
    return case


# ---- inputs, plain torch --------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _csr(m, src, dst):
    """Pull CSR of the edges src -> dst without self-loops and repeats: row offsets,
    ascending columns (sources), out-degrees."""
    keep = src != dst
    key = dst[keep] * m + src[keep]
    del src, dst, keep
    key = torch.unique(key)
    dst = torch.div(key, m, rounding_mode="floor")
    src = key - dst * m
    del key
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(dst, minlength=m), 0, out=rowptr[1:])
    outdeg = torch.bincount(src, minlength=m).to(torch.int32)
    return rowptr.to(torch.int32), src.to(torch.int32), outdeg


def _rmat(m, ef, seed):
    """RMAT graph of m vertices (draws past m are dropped), ids scrambled."""
    g = _generator(seed)
    bits = max(1, (m - 1).bit_length())
    a, b, c = RMAT
    parts, left = [], m * ef
    while left > 0:
        n = min(left, 1 << 25)
        left -= n
        s = torch.zeros(n, dtype=torch.int64, device=DEV)
        d = torch.zeros(n, dtype=torch.int64, device=DEV)
        for _ in range(bits):
            u = torch.rand(n, generator=g, device=DEV)
            s.mul_(2).add_(u >= a + b)
            d.mul_(2).add_(((u >= a) & (u < a + b)) | (u >= a + b + c))
        if m != 1 << bits:
            keep = (s < m) & (d < m)
            s, d = s[keep], d[keep]
        parts.append((s, d))
    perm = torch.randperm(m, generator=g, device=DEV)
    src = torch.cat([perm[s] for s, _ in parts])
    dst = torch.cat([perm[d] for _, d in parts])
    del parts, perm
    return _csr(m, src, dst)


def _batch_sizes(case):
    """Vertex offsets; the sizes belong to the case, the edges to the seed."""
    r = np.random.default_rng([case["graphs"], case["m_min"], case["m_max"]])
    lo, hi = math.log(case["m_min"]), math.log(case["m_max"])
    sizes = np.exp(r.uniform(lo, hi, case["graphs"])).astype(np.int64)
    return np.concatenate([[0], np.cumsum(sizes)])


def _batch(case, seed):
    """Block-diagonal pull graph: even graphs Erdos-Renyi (8 draws a vertex), odd ones
    Chung-Lu with degree exponent 2.1 (16 draws a vertex)."""
    g = _generator(seed)
    voff = _batch_sizes(case)
    m = int(voff[-1])
    off = torch.from_numpy(voff).to(DEV)
    size = off[1:] - off[:-1]
    odd = torch.arange(case["graphs"], device=DEV) % 2
    owner = torch.repeat_interleave(size * (8 + 8 * odd))
    # ranks scrambled within each graph, so that heavy vertices have any id
    vertex_owner = torch.repeat_interleave(size)
    order = torch.argsort(vertex_owner * (1 << 24)
                          + torch.randint(0, 1 << 24, (m,), generator=g, device=DEV))
    del vertex_owner
    share = 1.0 - 1.0 / (2.1 - 1.0)

    def ends():
        u = torch.rand(owner.numel(), generator=g, device=DEV, dtype=torch.float64)
        n = size[owner].double()
        heavy = (1.0 + u * ((n + 1.0) ** share - 1.0)) ** (1.0 / share) - 1.0
        v = torch.where(odd[owner] == 1, heavy, u * n).to(torch.int64)
        return order[torch.minimum(v, size[owner] - 1) + off[owner]]

    src = ends()
    dst = ends()
    return _csr(m, src, dst) + (voff.astype(np.int32),)


def _stencil(nx, ny, nz, seed):
    """27-point stencil with coefficients from the seed (off-diagonals in [-1.2, -0.8],
    a diagonal a little above the row's sum): row offsets, columns, values."""
    g = _generator(seed)
    n = nx * ny * nz
    i = torch.arange(n, device=DEV)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    cols, inside = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                inside.append((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
                              & (z + dz >= 0) & (z + dz < nz))
                cols.append((i + dx + nx * (dy + ny * dz)).to(torch.int32))
    col = torch.stack(cols, 1)
    ok = torch.stack(inside, 1)
    del cols, inside
    val = -0.8 - 0.4 * torch.rand((n, 27), generator=g, device=DEV)
    val[:, 13] = 0.0
    val[~ok] = 0.0
    val[:, 13] = 0.5 - val.sum(1)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(ok.sum(1), 0, out=rowptr[1:])
    return rowptr.to(torch.int32), col[ok].contiguous(), val[ok].contiguous()


def _colours(nx, ny, nz):
    """Rows by the parity colour of their point, and the colours' boundaries."""
    i = torch.arange(nx * ny * nz, device=DEV)
    colour = i % nx % 2 + 2 * ((i // nx) % ny % 2) + 4 * (i // (nx * ny) % 2)
    rows = torch.sort(colour, stable=True).indices.to(torch.int32)
    bounds = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV),
                        torch.cumsum(torch.bincount(colour, minlength=8), 0)])
    return rows, bounds.to(torch.int32).cpu().numpy()


def _values(n, seed, salt):
    g = _generator(seed * 31 + salt)
    return torch.randn(n, generator=g, device=DEV)


def _seeds(case, rowptr, outdeg, seed):
    """Seed vertices among those with in- and out-edges."""
    pool = torch.nonzero((rowptr[1:] > rowptr[:-1]) & (outdeg > 0)).flatten().cpu().numpy()
    r = np.random.default_rng(int(seed) * 104729 + 3)
    return r.choice(pool, case["k"], replace=len(pool) < case["k"]).astype(np.int32)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _blocked(case):
    return KEPT * case["ef"] * case["m"] >= BLOCKED_EDGES


def _limit(case):
    """Sweeps allowed: the reference's MAX_ITER at its default tolerance, else 100."""
    return 30 if case["tol"] >= 1e-3 else 100


# ---- one case -------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("call", "pull", "push", "noalloc", "ppr", "spmv_graph"):
        rowptr, col, outdeg = _rmat(case["m"], case["ef"], seed)
        m, nnz = case["m"], col.numel()
    if kind == "call":
        st.update(m=m, nnz=nnz, rowptr=rowptr.cpu().numpy(), col=col.cpu().numpy(),
                  outdeg=outdeg.cpu().numpy())
    elif kind in ("pull", "push", "ppr"):
        torch.cuda.synchronize()  # the library builds its layout on its own stream
        graph = G.Graph(rowptr, col, outdeg, m=m, nnz=nnz,
                        blocked=kind == "pull" and _blocked(case), push=kind == "push",
                        batched=kind == "ppr")
        graph.set_stream(_stream())
        st.update(graph=graph, m=m)
        if kind == "ppr":
            st["seeds"] = _seeds(case, rowptr, outdeg, seed)
            st["x"] = torch.empty((m, case["k"]), device=DEV)
        else:
            st["scores"] = torch.empty(m, device=DEV)
    elif kind == "noalloc":
        st.update(m=m, nnz=nnz, rowptr=rowptr, col=col, outdeg=outdeg,
                  scores=torch.empty(m, device=DEV))
    elif kind == "batch":
        rowptr, col, outdeg, voff = _batch(case, seed)
        torch.cuda.synchronize()
        graph = G.MultiGraph(rowptr, col, outdeg, voff, nnz=col.numel(),
                             blocked=col.numel() >= BLOCKED_EDGES)
        graph.set_stream(_stream())
        st.update(graph=graph, start=torch.from_numpy(graph.initial_scores()).to(DEV),
                  scores=torch.empty(int(voff[-1]), device=DEV))
    elif kind in ("spmv_stencil", "spmv_graph"):
        if kind == "spmv_stencil":
            rowptr, col, val = _stencil(case["nx"], case["ny"], case["nz"], seed)
        else:
            val = _values(col.numel(), seed, 3)
        m = rowptr.numel() - 1
        torch.cuda.synchronize()
        st.update(matrix=G.Matrix(rowptr, col, val, m=m, nnz=col.numel()),
                  x=_values(m, seed, 1), y=torch.empty(m, device=DEV))
    elif kind == "symgs":
        rowptr, col, val = _stencil(case["nx"], case["ny"], case["nz"], seed)
        rows, bounds = _colours(case["nx"], case["ny"], case["nz"])
        m = rowptr.numel() - 1
        torch.cuda.synchronize()
        st.update(smoother=G.SymGS(rowptr, col, val, rows, bounds, m=m, nnz=col.numel()),
                  x=torch.empty(m, device=DEV), b=_values(m, seed, 2))
    torch.cuda.synchronize()
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "call":
        m = st["m"]
        scores = np.full(m, np.float32(1.0) / np.float32(m), dtype=np.float32)
        G.PageRank(m, st["nnz"], st["rowptr"], st["col"], st["outdeg"], scores,
                   tol=case["tol"], max_iter=_limit(case))
        return {"scores": scores}
    if kind == "pull":
        st["scores"].fill_(1.0 / st["m"])
        st["graph"].pagerank(st["scores"], tol=case["tol"], max_iter=_limit(case))
        return {"scores": st["scores"]}
    if kind == "push":
        st["scores"].fill_(1.0 / st["m"])
        st["graph"].pagerank_push(st["scores"], tol=case["tol"], max_iter=_limit(case))
        return {"scores": st["scores"]}
    if kind == "noalloc":
        st["scores"].fill_(1.0 / st["m"])
        G.pagerank_noalloc(st["m"], st["nnz"], st["rowptr"], st["col"], st["outdeg"],
                           st["scores"], stream_handle=_stream(), tol=case["tol"],
                           max_iter=_limit(case))
        return {"scores": st["scores"]}
    if kind == "ppr":
        st["graph"].ppr(st["seeds"], out=st["x"], tol=case["tol"], max_iter=_limit(case))
        return {"x": st["x"]}
    if kind == "batch":
        st["scores"].copy_(st["start"])
        st["graph"].pagerank(st["scores"], tol=case["tol"], max_iter=_limit(case))
        return {"scores": st["scores"]}
    if kind in ("spmv_stencil", "spmv_graph"):
        st["y"].zero_()
        st["matrix"].spmv(st["x"], st["y"], _stream())
        return {"y": st["y"]}
    # the smoother runs on a stream of its own: x has to be there before the call
    st["x"].zero_()
    torch.cuda.current_stream().synchronize()
    st["smoother"].apply(st["x"], st["b"], sweeps=case["sweeps"])
    return {"x": st["x"]}


# ---- what a pass cannot do without ---------------------------------------------
def _sweeps(case):
    """Sweeps of a solve on an RMAT graph: about 12 for each power of ten."""
    return max(1, min(_limit(case), round(-12 * math.log10(case["tol"]) - 23)))


def _entries(case):
    """Entries of the 27-point matrix: each axis joins 3 n - 2 pairs."""
    return (3 * case["nx"] - 2) * (3 * case["ny"] - 2) * (3 * case["nz"] - 2)


def work(case):
    kind = case["kind"]
    if kind in ("call", "pull", "push", "noalloc"):
        m, nnz, n = case["m"], KEPT * case["ef"] * case["m"], _sweeps(case)
        return {"bytes": n * (4 * nnz + 28 * m), "flops": n * (nnz + 4 * m)}
    if kind == "ppr":
        m, nnz, k = case["m"], KEPT * case["ef"] * case["m"], case["k"]
        # a vector from a single seed stops after about half of a plain solve's sweeps
        n = max(1, round(-2 * math.log10(case["tol"])))
        return {"bytes": n * (4 * nnz + 8 * m + 16 * k * m), "flops": n * k * (nnz + 4 * m)}
    if kind == "batch":
        lo, hi = case["m_min"], case["m_max"]
        m = case["graphs"] * (hi - lo) / math.log(hi / lo)
        nnz = 10.2 * m
        n = 0.9 * _sweeps(case)
        return {"bytes": n * (4 * nnz + 28 * m), "flops": n * (nnz + 4 * m)}
    if kind == "spmv_graph":
        m, nnz = case["m"], KEPT * case["ef"] * case["m"]
        return {"bytes": 8 * nnz + 16 * m, "flops": 2 * nnz}
    m, nnz = case["nx"] * case["ny"] * case["nz"], _entries(case)
    if kind == "spmv_stencil":
        return {"bytes": 8 * nnz + 16 * m, "flops": 2 * nnz}
    # forward and backward over 8 colours; the turns repeat a colour, which sets the same x
    passes = case["sweeps"] * 14 + 1
    return {"bytes": passes / 8 * (8 * (nnz - m) + 16 * m), "flops": passes / 8 * 2 * nnz}


def tolerance(case):
    kind = case["kind"]
    if kind in ("spmv_stencil", "spmv_graph", "symgs"):
        # seen: 1e-7 against 64 bits; a row's terms have both signs
        return {"rel": 4e-7, "max": 1e-4}
    # 32-bit scores.  Seen against 64 bits: 1e-7 (pull, personalized), 2e-7 (push, whose
    # order of addition varies), 1e-6 (a hub's in-edges added one by one without
    # allocation); a vector or graph near its stop may take a sweep more or less.
    return {"rel": 4e-6, "max": 4e-4}


# ---- 64-bit answers in plain torch -------------------------------------------
def _sparse(rowptr, col, val, m):
    return torch.sparse_csr_tensor(rowptr.to(torch.int64), col.to(torch.int64), val, size=(m, m))


def _pagerank64(rowptr, col, outdeg, tol, limit, owner=None, sizes=None):
    """The recurrence in 64 bits.  With owner / sizes: each graph of a batch with its own
    base, residual and stop."""
    m = rowptr.numel() - 1
    A = _sparse(rowptr, col, torch.ones(col.numel(), dtype=torch.float64, device=DEV), m)
    deg = outdeg.clamp(min=1).double()
    if owner is None:
        s = torch.full((m,), 1.0 / m, dtype=torch.float64, device=DEV)
        for _ in range(limit):
            t = (1.0 - DAMP) / m + DAMP * (A @ (s / deg))
            r = float((t - s).abs().sum())
            s = t
            if r < tol:
                break
        return s
    n = sizes.numel()
    base = ((1.0 - DAMP) / sizes.double())[owner]
    s = (1.0 / sizes.double())[owner]
    going = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(limit):
        t = torch.where(going[owner], base + DAMP * (A @ (s / deg)), s)
        r = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, owner, (t - s).abs())
        s = t
        going &= r >= tol
        if not bool(going.any()):
            break
    return s


def _ppr64(rowptr, col, outdeg, seeds, tol, limit):
    m, k = rowptr.numel() - 1, len(seeds)
    A = _sparse(rowptr, col, torch.ones(col.numel(), dtype=torch.float64, device=DEV), m)
    deg = outdeg.clamp(min=1).double().unsqueeze(1)
    sink = outdeg == 0
    at = torch.from_numpy(seeds.astype(np.int64)).to(DEV)
    q = torch.arange(k, device=DEV)
    x = torch.zeros((m, k), dtype=torch.float64, device=DEV)
    x[at, q] = 1.0
    going = torch.ones(k, dtype=torch.bool, device=DEV)
    for _ in range(limit):
        t = (A @ (x / deg)).mul_(DAMP)
        t[at, q] += (1.0 - DAMP) + DAMP * x[sink].sum(0)
        r = (t - x).abs_().sum(0)
        x = torch.where(going, t, x)
        going &= r >= tol
        if not bool(going.any()):
            break
    return x


def _symgs64(case, rowptr, col, val, b):
    n = rowptr.numel() - 1
    rows, bounds = _colours(case["nx"], case["ny"], case["nz"])
    length = (rowptr[1:] - rowptr[:-1]).to(torch.int64)
    first = rowptr[:-1].to(torch.int64)
    lane = torch.arange(27, device=DEV)
    x = torch.zeros(n, dtype=torch.float64, device=DEV)
    b = b.double()
    order = list(range(8)) + list(range(7, -1, -1))
    for _ in range(case["sweeps"]):
        for c in order:
            r = rows[int(bounds[c]):int(bounds[c + 1])].to(torch.int64)
            ok = lane < length[r].unsqueeze(1)
            e = torch.where(ok, first[r].unsqueeze(1) + lane, 0)
            j = col[e].to(torch.int64)
            v = torch.where(ok, val[e].double(), 0.0)
            diag = torch.where(j == r.unsqueeze(1), v, 0.0).sum(1)
            off = torch.where(j == r.unsqueeze(1), 0.0, v * x[j]).sum(1)
            x[r] = (b[r] - off) / diag
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("call", "pull", "push", "noalloc"):
        rowptr, col, outdeg = _rmat(case["m"], case["ef"], seed)
        s = _pagerank64(rowptr, col, outdeg, case["tol"], _limit(case))
        return {"scores": s.cpu().numpy() if kind == "call" else s}
    if kind == "ppr":
        rowptr, col, outdeg = _rmat(case["m"], case["ef"], seed)
        return {"x": _ppr64(rowptr, col, outdeg, _seeds(case, rowptr, outdeg, seed),
                            case["tol"], _limit(case))}
    if kind == "batch":
        rowptr, col, outdeg, voff = _batch(case, seed)
        sizes = torch.from_numpy(np.diff(voff.astype(np.int64))).to(DEV)
        owner = torch.repeat_interleave(sizes)
        return {"scores": _pagerank64(rowptr, col, outdeg, case["tol"], _limit(case), owner,
                                      sizes)}
    if kind == "spmv_graph":
        rowptr, col, _ = _rmat(case["m"], case["ef"], seed)
        val = _values(col.numel(), seed, 3)
    else:
        rowptr, col, val = _stencil(case["nx"], case["ny"], case["nz"], seed)
    m = rowptr.numel() - 1
    if kind == "symgs":
        return {"x": _symgs64(case, rowptr, col, val, _values(m, seed, 2))}
    return {"y": _sparse(rowptr, col, val.double(), m) @ _values(m, seed, 1).double()}
