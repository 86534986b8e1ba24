"""Push-style PageRank (a scatter in source order into destination blocks, or edge by
edge with atomic float adds where a score is not finite) on the
GPU, held to the plain path's bar against the reference's pull recurrence
(1e-6 per vertex plus the reference's own float error on hub rows, sweeps
within one)."""
import numpy as np
import pytest

from graphs import degree_ladder, erdos_renyi, star

pytestmark = pytest.mark.gpu


def check(O, rp, col, od, s, it, tol, max_iter):
    ref, ref_it, _ = O.pr_plain_f32(rp, col, od, tol=tol, max_iter=max_iter)
    assert abs(it - ref_it) <= 1
    s64, _, _ = O.pr_f64(rp, col, od, tol=0.0, max_iter=it)
    assert np.all(np.abs(s - ref) <= 1e-6 + np.abs(ref - s64))


@pytest.mark.parametrize("maker", ["rmat", "er", "star", "ladder"])
def test_push_matches_reference(G, O, maker):
    rp, col, od = {"rmat": lambda: O.rmat_graph(15, 16, seed=3),
                   "er": lambda: erdos_renyi(20000, 8, seed=4),
                   "star": star, "ladder": degree_ladder}[maker]()
    # On the hub graphs the L1 residual's float rounding floor is about
    # m * ulp(score) ~ 1e-7; the tolerance sits well above it (as for the
    # pull solver's hub tests), where the arithmetic, not the rounding
    # noise of the atomic sums, decides the sweep count.
    tol = 1e-5 if maker in ("star", "ladder") else 1e-6
    with G.Graph(rp, col, od, push=True) as g:
        s, st = g.pagerank_push(tol=tol, max_iter=100)
        s2, st2 = g.pagerank_push(tol=tol, max_iter=100)
    check(O, rp, col, od, s, st.iterations, tol, 100)
    assert abs(st2.iterations - st.iterations) <= 1
    assert np.abs(s - s2).max() <= 1e-6


def test_push_caps_and_small_graphs(G, O):
    rp, col, od = O.rmat_graph(10, 8, seed=2)  # m < the shared-memory prefix
    with G.Graph(rp, col, od, push=True) as g:
        s, st = g.pagerank_push(tol=0.0, max_iter=5)
        assert st.iterations == 5
        check(O, rp, col, od, s, 5, 0.0, 5)
        s, st = g.pagerank_push(tol=1e-6, max_iter=0)
        assert st.iterations == 0
        assert np.all(s == np.float32(1.0) / np.float32(len(rp) - 1))


def test_push_needs_the_csr(G, O):
    rp, col, od = O.rmat_graph(8, 8, seed=1)
    with G.Graph(rp, col, od) as g:
        with pytest.raises(G.GprError) as e:
            g.pagerank_push()
        assert e.value.status == G.GPR_EUNSUPPORTED


def test_push_barrier_timeout(G, O):
    rp, col, od = O.rmat_graph(10, 8, seed=2)
    with G.Graph(rp, col, od, push=True) as g:
        o = G.options(tol=1e-6, max_iter=10, timeout_s=0.5)
        o.reserved[0] = 1
        with pytest.raises(G.GprError) as e:
            g.pagerank_push(opts=o)
        assert e.value.status == G.GPR_ETIMEOUT
        s, st = g.pagerank_push(tol=1e-6, max_iter=10)
        assert st.iterations > 0


@pytest.mark.parametrize("maker", ["rmat", "star", "no_edges", "one_edge"])
def test_push_in_blocks(G, O, maker):
    """The push solver's blocked solve gives the bits of the blocked pull solve on a
    layout built at creation, the same twice, and leaves the graph's own pull
    solves as they were."""
    rp, col, od = {"rmat": lambda: O.rmat_graph(13, 16, seed=5), "star": lambda: star(5000),
                   "no_edges": lambda: (np.zeros(301, np.int32), np.zeros(0, np.int32),
                                        np.zeros(300, np.int32)),
                   "one_edge": lambda: (np.array([0, 0, 1], np.int32), np.zeros(1, np.int32),
                                        np.array([1, 0], np.int32))}[maker]()
    kw = dict(tol=0.0, max_iter=6)
    with G.Graph(rp, col, od, blocked=True) as g:
        ref, _ = g.pagerank(form=G.FORM_BLOCKED, **kw)
    with G.Graph(rp, col, od, push=True) as g:
        before, _ = g.pagerank(**kw)
        a, st = g.pagerank_push(**kw)
        b, _ = g.pagerank_push(**kw)
        after, _ = g.pagerank(**kw)
    assert st.iterations == 6
    assert np.array_equal(a, ref) and np.array_equal(a, b)
    assert np.array_equal(before, after)


def test_push_non_finite_scores(G, O):
    """An infinite score cannot be held in fixed point: those edges add one by one, and
    the infinities reach the vertices that the reference's reach."""
    rp, col, od = erdos_renyi(3000, 6, seed=9)
    s0 = np.full(3000, np.float32(1 / 3000))
    s0[int(np.argmax(od))] = np.inf
    ref, _, _ = O.pr_plain_f32(rp, col, od, scores=s0, tol=0.0, max_iter=2)
    with G.Graph(rp, col, od, push=True) as g:
        g.pagerank_push(tol=0.0, max_iter=2)
        s, st = g.pagerank_push(s0.copy(), tol=0.0, max_iter=2)
    fin = np.isfinite(ref)
    assert st.iterations == 2 and not fin.all()
    assert np.array_equal(fin, np.isfinite(s))
    assert np.abs(s[fin] - ref[fin]).max() <= 1e-6


def far_start(kind, m, rp, col, od, O):
    """Finite starts whose largest score is far above 1/m."""
    rng = np.random.default_rng(len(kind))
    if kind == "one_vertex":
        s = np.zeros(m, dtype=np.float32)
        s[int(np.argmax(od))] = 1.0
    elif kind == "ones":
        s = np.ones(m, dtype=np.float32)
    elif kind == "random":
        s = rng.random(m).astype(np.float32)
    elif kind == "solution":
        s = O.pr_f64(rp, col, od, tol=1e-9, max_iter=200)[0].astype(np.float32)
    else:  # scores over some thirty binades, total 1
        w = np.exp(rng.normal(0, 6, m))
        s = (w / w.sum()).astype(np.float32)
    return s


def fp32_sweeps(rp, col, od, s0, sweeps):
    """The recurrence in FP64 and, per vertex, how far FP32 sweeps of any order of
    additions may be from it.  A sweep rounds a score's contribution, sum, product and
    update, 4 x 2^-24 relative, which may fall the same way for all (equal scores,
    the base) and is passed on as it is, d / outdeg of it; and the running sums of a row of k
    terms, 4 sqrt(k) 2^-24, which are independent from row to row and add in squares."""
    m = len(rp) - 1
    rows = np.repeat(np.arange(m), np.diff(rp))
    one, order = 4 * 2.0 ** -24, 4 * np.sqrt(np.diff(rp)) * 2.0 ** -24
    deg = np.maximum(od, 1).astype(np.float64)
    d = float(np.float32(0.85))
    s, lin, var = s0.astype(np.float64), np.zeros(m), np.zeros(m)
    for _ in range(sweeps):
        s = (1.0 - d) / m + d * np.bincount(rows, (s / deg)[col], minlength=m)
        lin = one * s + d * np.bincount(rows, (lin / deg)[col], minlength=m)
        var = (order * s) ** 2 + d * d * np.bincount(rows, (var / deg ** 2)[col], minlength=m)
    return s, lin + np.sqrt(var)


@pytest.mark.parametrize("kind", ["one_vertex", "ones", "random", "solution", "wide"])
def test_push_from_starts_far_from_uniform(G, O, kind):
    """The precision of FP32 sweeps whatever the finite start, and their sweep count."""
    rp, col, od = O.rmat_graph(17, 16, seed=6)
    m = len(rp) - 1
    s0 = far_start(kind, m, rp, col, od, O)
    with G.Graph(rp, col, od, push=True) as g:
        s, st = g.pagerank_push(s0.copy(), tol=0.0, max_iter=20)
        t, st_t = g.pagerank_push(s0.copy(), tol=1e-5, max_iter=200)
    ref, off = fp32_sweeps(rp, col, od, s0, 20)
    assert st.iterations == 20
    assert np.all(np.abs(s - ref) <= off), np.max(np.abs(s - ref) / off)
    _, n, _ = O.pr_f64(rp, col, od, tol=1e-5, max_iter=200, init=s0)
    assert abs(st_t.iterations - n) <= 1


def test_push_with_too_small_out_degrees(G, O):
    """Out-degrees are the caller's.  Half of the edges' number lets the scores grow in
    every sweep, past what fixed point holds (2^55 here), and 0 gives infinities:
    both as the reference's recurrence has them."""
    rp, col, od = O.rmat_graph(12, 16, seed=7)
    m = len(rp) - 1
    half = np.where(od > 1, od // 2, od).astype(np.int32)
    with G.Graph(rp, col, half, push=True) as g:
        s, st = g.pagerank_push(tol=0.0, max_iter=80)
    ref, _, _ = O.pr_f64(rp, col, half, tol=0.0, max_iter=80)
    assert ref.max() > 2.0 ** 40
    # 80 sweeps of (8 + 4 sqrt(k)) 2^-24 per vertex, passed on from sweep to sweep
    bound = 80 * (8 + 4 * np.sqrt(np.diff(rp).max())) * 2.0 ** -24
    assert np.all(np.abs(s - ref) <= bound * ref)
    none = od.copy()
    none[int(np.argmax(od))] = 0
    with G.Graph(rp, col, none, push=True) as g:
        s, st = g.pagerank_push(tol=0.0, max_iter=2)
    ref, _, _ = O.pr_plain_f32(rp, col, none, tol=0.0, max_iter=2)
    fin = np.isfinite(ref)
    assert 0 < np.count_nonzero(fin) < m
    assert np.array_equal(fin, np.isfinite(s))
    assert np.abs(s[fin] - ref[fin]).max() <= 1e-6


@pytest.mark.parametrize("maker", ["rmat", "er", "star", "ladder"])
def test_push_edge_by_edge(G, O, maker):
    """The form without blocks, which one vertex with an edge more than its out-degree
    says selects: the reference's recurrence with that degree, its stop rule, sweep
    caps and the bounded wait at its barrier."""
    rp, col, od = {"rmat": lambda: O.rmat_graph(15, 16, seed=3),
                   "er": lambda: erdos_renyi(20000, 8, seed=4),
                   "star": star, "ladder": degree_ladder}[maker]()
    od = od.copy()
    some = np.flatnonzero(od > 1)
    od[some[np.argmin(np.diff(rp)[some])]] -= 1  # of few in-edges: the scores stay bounded
    tol = 1e-5 if maker in ("star", "ladder") else 1e-6
    with G.Graph(rp, col, od, push=True) as g:
        s, st = g.pagerank_push(tol=tol, max_iter=100)
        t, st_t = g.pagerank_push(tol=0.0, max_iter=5)
        z, st_z = g.pagerank_push(tol=tol, max_iter=0)
        o = G.options(tol=tol, max_iter=10, timeout_s=0.5)
        o.reserved[0] = 1
        with pytest.raises(G.GprError) as e:
            g.pagerank_push(opts=o)
        again, st_a = g.pagerank_push(tol=tol, max_iter=100)
    assert e.value.status == G.GPR_ETIMEOUT
    m = len(rp) - 1
    s0 = np.full(m, np.float32(1.0) / np.float32(m))
    _, n, _ = O.pr_f64(rp, col, od, tol=tol, max_iter=100)
    assert abs(st.iterations - n) <= 1 and abs(st_a.iterations - n) <= 1
    assert st_t.iterations == 5 and st_z.iterations == 0 and np.array_equal(z, s0)
    for got, sweeps in ((s, st.iterations), (again, st_a.iterations), (t, 5)):
        ref, off = fp32_sweeps(rp, col, od, s0, sweeps)
        assert np.all(np.abs(got - ref) <= off), np.max(np.abs(got - ref) / off)
    # the scores in, all sweeps, the scores out: the blocked solve has one launch more
    assert st.gpu_launches == 3
