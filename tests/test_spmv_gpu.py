"""CSR SpMV on the GPU through the C ABI, checked against the oracle.

Rows with at most 64 entries are summed with the reference's float
operations in the reference's order (src/spmv/omp_base.cc:18-28): the result
must be bit-identical.  Longer rows are summed as a tree: their error is
bounded by 1e-6 of the sum of |products|.  The 27-point stencil at full size
(128^3, 55.7M nonzeros) is checked bit-for-bit, which also meets the
reference verifier's maximum-relative-error criterion (<= 1e-6 here).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stencil_small_bit_identical(G, O):
    Ap, Aj, Ax = O.stencil27(20)
    m = len(Ap) - 1
    x = O.uniform_f32(m, 5)
    for y0 in (np.zeros(m, np.float32), O.uniform_f32(m, 6)):
        y = y0.copy()
        G.SpmvSolver(m, len(Aj), Ap, Aj, Ax, x, y)
        assert np.array_equal(y, O.spmv_f32(Ap, Aj, Ax, x, y0))


def test_stencil_128_full_size(G, O):
    torch = pytest.importorskip("torch")
    A = G.gen_stencil27(128)
    assert A.m == 128 ** 3 and A.nnz == 382 ** 3
    x = torch.empty(A.m, dtype=torch.float32, device="cuda")
    G.gen_uniform(A.m, 11, x)
    y = torch.zeros(A.m, dtype=torch.float32, device="cuda")
    M = G.Matrix(A.rowptr, A.col, A.third, m=A.m, nnz=A.nnz)
    M.spmv(x, y)
    torch.cuda.synchronize()
    Ap, Aj, Ax = A.rowptr.to_numpy(), A.col.to_numpy(), A.third.to_numpy()
    xr = O.uniform_f32(A.m, 11)
    assert np.array_equal(x.cpu().numpy(), xr)
    yr = O.spmv_f32(Ap, Aj, Ax, xr, np.zeros(A.m, np.float32))
    yg = y.cpu().numpy()
    assert O.max_rel_err(yg, yr) <= 1e-6
    assert np.array_equal(yg, yr)
    M.close()
    A.close()


def test_long_and_ragged_rows(G, O):
    rng = np.random.default_rng(2)
    m = 3000
    lens = rng.integers(0, 20, m)
    lens[[0, 7, 100, 2999]] = [5000, 65, 64, 3000]
    lens[[1, 2]] = 0
    Ap = np.zeros(m + 1, np.int32)
    np.cumsum(lens, out=Ap[1:])
    Aj = np.concatenate([np.sort(rng.choice(m, size=l, replace=l > m)) for l in lens]).astype(np.int32)
    Ax = (1.0 - 2.0 * rng.random(len(Aj))).astype(np.float32)
    x = rng.random(m).astype(np.float32)
    y0 = rng.random(m).astype(np.float32)
    y = y0.copy()
    G.SpmvSolver(m, len(Aj), Ap, Aj, Ax, x, y)
    yr = O.spmv_f32(Ap, Aj, Ax, x, y0)
    short = lens <= 64
    assert np.array_equal(y[short], yr[short])
    absum = np.array([np.abs(x[Aj[Ap[i]:Ap[i + 1]]] * Ax[Ap[i]:Ap[i + 1]]).sum() + abs(y0[i])
                      for i in range(m)])
    assert np.all(np.abs(y - yr) <= 1e-6 * absum + 1e-30)


def test_empty_matrix(G):
    Ap = np.zeros(11, np.int32)
    y = np.arange(10, dtype=np.float32)
    G.SpmvSolver(10, 0, Ap, np.array([], np.int32), np.array([], np.float32),
                 np.ones(10, np.float32), y)
    assert np.array_equal(y, np.arange(10, dtype=np.float32))


@pytest.mark.parametrize("m", [1, 1023, 1024, 1025, 40000])
@pytest.mark.parametrize("hot", [False, True])
def test_ragged_matrix(G, O, m, hot):
    """Ragged row lengths (windows of 1024 rows sorted by length), a matrix smaller than
    a window and one row short of and past it, columns skewed (at 40,000 rows enough
    for 1024 of them to be staged; test_spmv_columns_are_staged pins the count) or
    uniform; empty rows, lengths around a lane's row (64), a
    chunk's round (384) and a chunk (4096).  Short rows are the oracle's bits."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(m + hot)
    lens = np.minimum(rng.zipf(1.6, m) - 1, 60)
    edge = [63, 64, 65, 383, 384, 385, 4095, 4096, 4097, 9000, 0, 1, 12, 13]
    for i, d in enumerate(edge):
        if i < m:
            lens[(i * 71) % m] = d
    Ap = np.zeros(m + 1, np.int32)
    np.cumsum(lens, out=Ap[1:])
    n = int(Ap[-1])
    Aj = (m * rng.random(n) ** (6 if hot else 1)).astype(np.int32)
    Ax = rng.standard_normal(n).astype(np.float32)
    x = rng.standard_normal(m).astype(np.float32)
    y0 = rng.standard_normal(m).astype(np.float32)
    ref = O.spmv_f32(Ap, Aj, Ax, x, y0)
    A = G.Matrix(Ap, Aj, Ax)
    dx, y = torch.from_numpy(x).cuda(), torch.from_numpy(y0.copy()).cuda()
    A.spmv(dx, y, torch.cuda.current_stream().cuda_stream)
    got = y.cpu().numpy()
    A.close()
    once = y0.copy()
    G.SpmvSolver(m, n, Ap, Aj, Ax, x, once)
    absum = np.abs(y0).astype(np.float64)
    np.add.at(absum, np.repeat(np.arange(m), lens), np.abs(x[Aj] * Ax))
    for out in (got, once):
        assert np.array_equal(out[lens <= 64], ref[lens <= 64])
        assert np.all(np.abs(out - ref) <= 1e-6 * absum + 1e-30)


@pytest.mark.parametrize("k,rows,ragged", [(65, 3000, False), (100, 2000, False), (636, 500, False),
                                           (640, 500, True), (1000, 4736, True),
                                           (1000, 4737, False), (9000, 40, True)])
@pytest.mark.parametrize("short", [0, 5000])
def test_evenly_long_rows(G, O, k, rows, ragged, short):
    """Rows of k entries each, and `short` rows of 3: natural order unless a chunk (of at
    most 4096 entries) has 640 entries and a warp's share of all (148 SMs x 32 warps);
    either way every row is within 1e-6 of its absolute sum of the oracle's."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(k)
    lens = np.concatenate([np.full(rows, k), np.full(short, 3)])
    m = len(lens)
    Ap = np.zeros(m + 1, np.int32)
    np.cumsum(lens, out=Ap[1:])
    n = int(Ap[-1])
    Aj = rng.integers(0, m, n).astype(np.int32)
    Ax = rng.standard_normal(n).astype(np.float32)
    x = rng.standard_normal(m).astype(np.float32)
    y0 = rng.standard_normal(m).astype(np.float32)
    A = G.Matrix(Ap, Aj, Ax)
    if short and rows == 4736:  # the short rows' entries take it past the share
        ragged = False
    assert A.layout()["n_slices"] == (-(-m // 1024) * 32 if ragged else -(-m // 32))
    dx, y = torch.from_numpy(x).cuda(), torch.from_numpy(y0.copy()).cuda()
    torch.cuda.synchronize()
    A.spmv(dx, y, torch.cuda.current_stream().cuda_stream)
    got = y.cpu().numpy()
    A.close()
    ref = O.spmv_f32(Ap, Aj, Ax, x, y0)
    absum = np.abs(y0).astype(np.float64)
    np.add.at(absum, np.repeat(np.arange(m), lens), np.abs(x[Aj] * Ax))
    assert np.array_equal(got[lens <= 64], ref[lens <= 64])
    assert np.all(np.abs(got - ref) <= 1e-6 * absum + 1e-30)
