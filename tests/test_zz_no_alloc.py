"""The PageRank entry point that allocates nothing (gpr_pagerank_noalloc).

Callers whose device memory is owned by their own allocator, or that may not
take the synchronisation a cudaMalloc / cudaFree can cause, need a solver that
allocates no memory.  gpr_pagerank_noalloc keeps its scratch in a fixed device
array inside the library; this test calls it through the C ABI on device
arrays, twice in a row (the second call reuses the array the first one left
behind), and checks each result against the existing entry point
(gpr_graph_create + gpr_pagerank) within the tolerance the other PageRank
tests use: 1e-6 absolute per vertex and the same sweep count within one.
Its sweep sums each row in CSR order with the reference's float operations,
so its scores are also compared bit for bit with the oracle's restatement of
the reference's OpenMP solver (src/pr/omp_base.cc:9-49).  Malformed CSR input
is rejected with GPR_EINVAL.  This file is collected last so that a run
stopping at the first failure has already run every other test.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ABS_TOL = 1e-6


def test_noalloc_matches_existing_entry_point_twice(G, O):
    torch = pytest.importorskip("torch")
    rp, col, od = O.rmat_graph(15, 16, seed=21)
    m, nnz = len(rp) - 1, len(col)
    with G.Graph(rp, col, od) as g:
        ref, st_ref = g.pagerank(tol=1e-6, max_iter=100)
    d_rp = torch.from_numpy(rp).cuda()
    d_col = torch.from_numpy(col).cuda()
    d_od = torch.from_numpy(od).cuda()
    for call in range(2):
        d_s = torch.full((m,), float(np.float32(1.0) / np.float32(m)), dtype=torch.float32,
                         device="cuda")
        st = G.pagerank_noalloc(m, nnz, d_rp, d_col, d_od, d_s, tol=1e-6, max_iter=100)
        s = d_s.cpu().numpy()
        assert abs(st.iterations - st_ref.iterations) <= 1, (call, st.iterations, st_ref.iterations)
        assert np.abs(s - ref).max() <= ABS_TOL, call


def test_noalloc_is_bit_identical_to_the_oracle(G, O):
    torch = pytest.importorskip("torch")
    rp, col, od = O.rmat_graph(14, 16, seed=5)
    m, nnz = len(rp) - 1, len(col)
    d_rp, d_col, d_od = (torch.from_numpy(a).cuda() for a in (rp, col, od))
    for tol, max_iter in ((1e-4, 100), (0.0, 7)):
        d_s = torch.full((m,), float(np.float32(1.0) / np.float32(m)), dtype=torch.float32,
                         device="cuda")
        st = G.pagerank_noalloc(m, nnz, d_rp, d_col, d_od, d_s, tol=tol, max_iter=max_iter)
        ref, n_ref, _ = O.pr_plain_f32(rp, col, od, tol=tol, max_iter=max_iter)
        assert abs(st.iterations - n_ref) <= 1, (st.iterations, n_ref)
        if st.iterations != n_ref:  # residual within rounding of tol: same sweeps as the GPU
            ref, _, _ = O.pr_plain_f32(rp, col, od, tol=0.0, max_iter=st.iterations)
        assert np.array_equal(d_s.cpu().numpy(), ref), (tol, max_iter)


@pytest.mark.parametrize("case", ["column_out_of_range", "last_offset", "decreasing",
                                  "negative_degree", "edges_without_vertices"])
@pytest.mark.parametrize("max_iter", [30, 0])
def test_noalloc_rejects_malformed_csr(G, case, max_iter):
    torch = pytest.importorskip("torch")
    rp = np.array([0, 2, 3, 5], dtype=np.int32)
    col = np.array([1, 2, 0, 0, 1], dtype=np.int32)
    od = np.array([2, 2, 1], dtype=np.int32)
    m, nnz = 3, 5
    if case == "column_out_of_range":
        col[3] = 3
    elif case == "last_offset":
        rp[3] = 4
    elif case == "decreasing":
        rp[1], rp[2] = 3, 2
    elif case == "negative_degree":
        od[1] = -1
    else:
        m = 0
    d = [torch.from_numpy(a).cuda() for a in (rp, col, od)]
    d_s = torch.full((3,), 1.0 / 3, dtype=torch.float32, device="cuda")
    with pytest.raises(G.GprError) as e:
        G.pagerank_noalloc(m, nnz, d[0], d[1], d[2], d_s, tol=1e-4, max_iter=max_iter)
    assert e.value.status == G.GPR_EINVAL


def test_noalloc_rejects_sizes_beyond_its_scratch(G):
    limit = G.pagerank_noalloc_max_vertices()
    assert limit == 1 << 20
    with pytest.raises(G.GprError) as e:
        G.pagerank_noalloc(limit + 1, 0, 1, 1, 1, 1)
    assert e.value.status == G.GPR_EINVAL and "limit" in str(e.value)


@pytest.mark.parametrize("hub,deg", [(0, 1), (255, 4095), (256, 4096), (300, 4097), (9999, 9998)])
def test_noalloc_long_rows_at_tile_edges(G, O, hub, deg):
    """A row as long as the staged tile, one edge shorter and longer, and longer
    than two tiles, at the first, last and an inner row of a CTA: every score
    equals the oracle's bit for bit (the same float additions in CSR order)."""
    torch = pytest.importorskip("torch")
    from graphs import in_csr
    rng = np.random.default_rng(hub + deg)
    m = 10000
    src = rng.choice(np.delete(np.arange(m), hub), deg, replace=False)
    more = rng.integers(0, m, (2, 3 * m))
    more = more[:, more[1] != hub]
    rp, col, od = in_csr(m, np.concatenate([src, more[0]]),
                         np.concatenate([np.full(deg, hub), more[1]]))
    assert rp[hub + 1] - rp[hub] == deg
    d_rp, d_col, d_od = (torch.from_numpy(a).cuda() for a in (rp, col, od))
    d_s = torch.full((m,), float(np.float32(1.0) / np.float32(m)), device="cuda")
    G.pagerank_noalloc(m, len(col), d_rp, d_col, d_od, d_s, tol=0.0, max_iter=4)
    ref, _, _ = O.pr_plain_f32(rp, col, od, tol=0.0, max_iter=4)
    assert np.array_equal(d_s.cpu().numpy(), ref)


@pytest.mark.parametrize("kind", ["uniform", "equal", "halves", "zeros", "wide", "tiny", "negative",
                                  "infinite"])
def test_noalloc_long_rows_add_in_order(G, O, kind):
    """Long rows are added by a warp as integers within a binade where that gives
    what the additions in CSR order give; whatever the values (ties, zeros, sums
    that leave their binade at once, denormal, negative and infinite ones), the
    scores are the oracle's bits."""
    torch = pytest.importorskip("torch")
    from graphs import in_csr
    rng = np.random.default_rng(len(kind))
    m, hubs = 12000, 40
    counts = rng.integers(200, 9000, hubs)
    src = np.concatenate([rng.choice(m, n, replace=False) for n in counts]
                         + [rng.integers(0, m, 4 * m)])
    dst = np.concatenate([np.repeat(np.arange(hubs) * 7, counts), rng.integers(0, m, 4 * m)])
    rp, col, od = in_csr(m, src, dst)
    s0 = rng.random(m).astype(np.float32)
    if kind == "equal":
        s0 = np.full(m, 1.0 / m, dtype=np.float32)
    elif kind == "halves":
        s0 = (rng.integers(0, 64, m) / 64 * od).astype(np.float32)
    elif kind == "zeros":
        s0[rng.random(m) < 0.7] = 0.0
    elif kind == "wide":
        s0 = np.exp(rng.normal(0, 18, m)).astype(np.float32)
    elif kind == "tiny":
        s0 *= np.float32(1e-38)
    elif kind == "negative":
        s0 -= np.float32(0.5)
    elif kind == "infinite":
        s0[m // 2] = np.inf
    d_rp, d_col, d_od = (torch.from_numpy(a).cuda() for a in (rp, col, od))
    d_s = torch.from_numpy(s0.copy()).cuda()
    G.pagerank_noalloc(m, len(col), d_rp, d_col, d_od, d_s, tol=0.0, max_iter=3)
    ref, _, _ = O.pr_plain_f32(rp, col, od, scores=s0, tol=0.0, max_iter=3)
    assert np.array_equal(d_s.cpu().numpy(), ref, equal_nan=True)
