"""What entry points do when one of their device allocations fails: the call falls back
or reports it, keeps no block that it cannot use, and the next call works; and what
they owe to a block that held other data; and what only the size of an allocation
shows.  Each case runs in a process of its own with
alloc_shim.cc ahead of the library; the failure is a status on the host."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PRELUDE = """
import ctypes, os, sys
shim = ctypes.CDLL(sys.argv[1], ctypes.RTLD_GLOBAL)
sys.path[:0] = [sys.argv[2], os.path.join(sys.argv[2], "tests")]
import numpy as np
import gardenia_ocl_b200 as G
import oracle as O
from graphs import erdos_renyi

def fail(what, status, count=1):
    shim.shim_fail(what.encode(), status, count)

shim.shim_bytes.restype = ctypes.c_longlong

what, status = sys.argv[3], int(sys.argv[4])
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shim") / "alloc_shim.so")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", out,
                    os.path.join(ROOT, "tests", "alloc_shim.cc"), "-ldl"], check=True)
    return out


def run(shim, body, what, status):
    p = subprocess.run([sys.executable, "-c", PRELUDE + body, shim, ROOT, what, str(status)],
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    assert p.stdout.splitlines()[-1] == "done"


PUSH = """
rp, col, od = O.rmat_graph(13, 16, seed=5)
with G.Graph(rp, col, od, push=True) as g:
    ref, _ = g.pagerank_push(tol=0.0, max_iter=6)
before = shim.shim_live()
g = G.Graph(rp, col, od, push=True)
made = shim.shim_live()
fail(what, status)
if status == G.GPR_ENOMEM:  # edge by edge: sources, destinations and sums are kept, no blocks
    s, st = g.pagerank_push(tol=0.0, max_iter=6)
    assert shim.shim_live() == made + 3, (shim.shim_live(), made)
else:  # reported; nothing kept; the next call builds again
    try:
        g.pagerank_push(tol=0.0, max_iter=6)
        raise SystemExit("no error")
    except G.GprError as e:
        assert e.status == status
    assert shim.shim_live() == made, (shim.shim_live(), made)
    s, st = g.pagerank_push(tol=0.0, max_iter=6)
    assert np.array_equal(s, ref)
assert shim.shim_pending() == 0
assert st.iterations == 6 and np.abs(s - ref).max() <= 1e-6
a, _ = g.pagerank(tol=0.0, max_iter=6)
assert np.abs(a - ref).max() <= 1e-6
g.close()
assert shim.shim_live() == before, (shim.shim_live(), before)
print("done")
"""


@pytest.mark.parametrize("what", ["identity", "largest score", "score sums", "cta residuals"])
@pytest.mark.parametrize("status", ["GPR_ENOMEM", "GPR_ECUDA"])
def test_push_layout(G, shim, what, status):
    run(shim, PUSH, what, getattr(G, status))


SPMV = """
import torch
rng = np.random.default_rng(3)
m = 60000
lens = np.minimum(rng.zipf(1.6, m) - 1, 3000)
Ap = np.zeros(m + 1, np.int32)
np.cumsum(lens, out=Ap[1:])
n = int(Ap[-1])
Aj = (m * rng.random(n) ** 8).astype(np.int32)  # columns worth staging
Ax = rng.standard_normal(n).astype(np.float32)
x = rng.standard_normal(m).astype(np.float32)
ref = O.spmv_f32(Ap, Aj, Ax, x, np.zeros(m, np.float32))
absum = np.zeros(m)
np.add.at(absum, np.repeat(np.arange(m), lens), np.abs(x[Aj] * Ax))
before = shim.shim_live()
fail(what, status)
if status == G.GPR_ENOMEM:
    A = G.Matrix(Ap, Aj, Ax)
else:
    try:
        G.Matrix(Ap, Aj, Ax)
        raise SystemExit("no error")
    except G.GprError as e:
        assert e.status == status
    assert shim.shim_live() == before, (shim.shim_live(), before)
    A = G.Matrix(Ap, Aj, Ax)
assert shim.shim_pending() == 0
dx, y = torch.from_numpy(x).cuda(), torch.zeros(m, device="cuda")
torch.cuda.synchronize()
A.spmv(dx, y, torch.cuda.current_stream().cuda_stream)
got = y.cpu().numpy()
A.close()
assert shim.shim_live() == before, (shim.shim_live(), before)
assert np.array_equal(got[lens <= 64], ref[lens <= 64])
assert np.all(np.abs(got - ref) <= 1e-6 * absum + 1e-30)
print("done")
"""


@pytest.mark.parametrize("what", ["column counts", "hot columns", "hot column index"])
@pytest.mark.parametrize("status", ["GPR_ENOMEM", "GPR_ECUDA"])
def test_spmv_staged_columns(G, shim, what, status):
    """Without room for the search of columns to stage, the matrix does without."""
    run(shim, SPMV, what, getattr(G, status))


@pytest.mark.parametrize("what", ["slot lengths", "slot rows", "slice lines"])
@pytest.mark.parametrize("status", ["GPR_ENOMEM", "GPR_ECUDA"])
def test_spmv_slots(G, shim, what, status):
    """Without room for sorted rows, a ragged matrix keeps its rows in natural order."""
    run(shim, SPMV, what, getattr(G, status))


FIRST_MULTIPLY = """
import torch
rng = np.random.default_rng(5)
m = 20000
lens = np.full(m, 4)
lens[:40] = 9000  # three chunks a row
Ap = np.zeros(m + 1, np.int32)
np.cumsum(lens, out=Ap[1:])
n = int(Ap[-1])
Aj = rng.integers(0, m, n).astype(np.int32)
Ax = rng.standard_normal(n).astype(np.float32)
x = rng.standard_normal(m).astype(np.float32)
ref = O.spmv_f32(Ap, Aj, Ax, x, np.zeros(m, np.float32))
absum = np.zeros(m)
np.add.at(absum, np.repeat(np.arange(m), lens), np.abs(x[Aj] * Ax))
side = torch.cuda.Stream()
dx = torch.from_numpy(x).cuda()
ys = [torch.zeros(m, device="cuda") for _ in range(3)]
ones = np.ones(128, np.int32)
blocks = [ctypes.c_void_p() for _ in range(4)]
for p in blocks:
    assert G.lib().gpr_malloc(ctypes.byref(p), 512) == 0
    assert G.lib().gpr_memcpy(p, ctypes.c_void_p(ones.ctypes.data), 512) == 0
torch.cuda.synchronize()
for p in blocks:
    G.lib().gpr_free(p)
# what the default stream does behind the counters' allocation comes late
late = ctypes.CFUNCTYPE(None)(lambda: torch.cuda._sleep(40000000))
shim.shim_call(what.encode(), late)
A = G.Matrix(Ap, Aj, Ax)
shim.shim_call(b"", ctypes.CFUNCTYPE(None)())
for y in ys:
    A.spmv(dx, y, side.cuda_stream)
side.synchronize()
torch.cuda.synchronize()
for y in ys:
    assert np.all(np.abs(y.cpu().numpy() - ref) <= 1e-6 * absum + 1e-30)
A.close()
print("done")
"""


def test_spmv_first_multiply_on_a_stream_of_its_own(G, shim):
    """The arrival counters are clear before gpr_matrix_create returns: the first
    multiply on a stream that waits for no other finds them so."""
    run(shim, FIRST_MULTIPLY, "spmv counters", 0)


STAGED = """
import torch
want, spread = int(what), status  # columns to be staged, and entries beside the limit
m = 1000000 if want <= 1024 else 300000
n = 4000000 if want <= 1024 else 8000000
rng = np.random.default_rng(want + spread)
lens = np.minimum(rng.zipf(1.5, m), 5000)
while lens.sum() < n:
    lens[rng.integers(0, m, 1000)] += 1
over = int(lens.sum() - n)
for r in np.argsort(-lens):  # down to n entries in all
    cut = min(over, int(lens[r]) - 1)
    lens[r] -= cut
    over -= cut
    if not over:
        break
Ap = np.zeros(m + 1, np.int32)
np.cumsum(lens, out=Ap[1:])
assert Ap[-1] == n
top = 1024 if want <= 1024 else want
if want <= 1024:  # exactly the limit (n / 16 and 148 loads a column), and `spread` more
    hot = n // 16 + 148 * top + spread
    cols = np.concatenate([np.arange(hot) % top, rng.integers(top, m, n - hot)])
else:
    cols = np.concatenate([np.arange(400 * top) % top, rng.integers(top, m, n - 400 * top)])
Aj = (rng.permutation(m)[rng.permutation(cols)]).astype(np.int32)
Ax = rng.standard_normal(n).astype(np.float32)
x = rng.standard_normal(m).astype(np.float32)
A = G.Matrix(Ap, Aj, Ax)
assert A.layout()["n_slices"] == -(-m // 1024) * 32  # the ragged layout
assert shim.shim_bytes(b"hot columns") == 4 * want, shim.shim_bytes(b"hot columns")
dx, y = torch.from_numpy(x).cuda(), torch.zeros(m, device="cuda")
torch.cuda.synchronize()
A.spmv(dx, y, torch.cuda.current_stream().cuda_stream)
got = y.cpu().numpy()
A.close()
ref = O.spmv_f32(Ap, Aj, Ax, x, np.zeros(m, np.float32))
absum = np.bincount(np.repeat(np.arange(m), lens), np.abs(x[Aj] * Ax), minlength=m)
assert np.array_equal(got[lens <= 64], ref[lens <= 64])
assert np.all(np.abs(got - ref) <= 1e-6 * absum + 1e-30)
print("done")
"""


@pytest.mark.parametrize("want,spread", [(0, 0), (1024, 1), (16384, 0)])
def test_spmv_columns_are_staged(G, shim, want, spread):
    """Columns are staged where their entries, less the 148 loads a column, are over 1/16
    of all: none at the limit, 1024 with an entry more, and as many as fit (16384,
    64 KB) where that many are frequent; short rows are the oracle's bits."""
    run(shim, STAGED, str(want), spread)
