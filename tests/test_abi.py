"""The C-ABI library loads and exports every symbol include/*.h declares;
without a GPU every entry point reports ENODEV instead of crashing."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT, has_gpu

HEADERS = ["gpr.h", "gardenia_pr.h", "gardenia_spmv.h", "gardenia_symgs.h", "gardenia_graph_io.h"]


def declared_c_functions():
    src = open(os.path.join(ROOT, "include", "gpr.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(gpr_\w+)\s*\(", src)))


def exported(lib_path):
    out = subprocess.run(["nm", "-D", "--defined-only", lib_path], capture_output=True,
                         text=True, check=True).stdout
    return {l.split()[-1] for l in out.splitlines() if " T " in l}


def test_every_declared_c_symbol_is_exported(G):
    names = declared_c_functions()
    assert len(names) >= 25
    syms = exported(G.LIB_PATH)
    missing = [n for n in names if n not in syms]
    assert not missing, missing


def test_cpp_dropins_exported_with_reference_mangling(G):
    # The reference's own symbols (C++ linkage, src/pr/pr.h:23-24,
    # src/spmv/spmv.h:29-30, src/symgs/symgs.h:28-29, include/graph_io.h:280).
    syms = exported(G.LIB_PATH)
    for s in ["_Z8PRSolveriiPiS_S_S_S_Pf", "_Z10PRVerifieriPiS_S_S_S_Pfd",
              "_Z8PageRankiiPiS_S_Pf", "_Z10SpmvSolveriiPiS_PfS0_S0_",
              "_Z12SpmvVerifieriiPiS_PfS0_S0_S0_", "_Z10read_graphiPPcRiS1_S1_RPiS3_S3_RPfbbbbb",
              "_Z11SymGSSolveriiPiS_S_PfS0_S0_St6vectorIiSaIiEE",
              "_Z13SymGSVerifieriPiS_S_PfS0_S0_S0_St6vectorIiSaIiEE"]:
        assert s in syms, s


def test_headers_compile_as_cpp():
    src = "".join(f'#include "{h}"\n' for h in HEADERS + ["gardenia_timer.h"]) + "int main(){return 0;}\n"
    p = subprocess.run(["/usr/bin/g++", "-std=c++17", "-fsyntax-only", "-x", "c++", "-",
                        "-I", os.path.join(ROOT, "include")], input=src, text=True,
                       capture_output=True)
    assert p.returncode == 0, p.stderr


def test_c_header_compiles_as_c():
    src = '#include "gpr.h"\nint main(void){gpr_pr_opts o; return gpr_pr_opts_default(&o);}\n'
    p = subprocess.run(["/usr/bin/gcc", "-std=c99", "-fsyntax-only", "-x", "c", "-",
                        "-I", os.path.join(ROOT, "include")], input=src, text=True,
                       capture_output=True)
    assert p.returncode == 0, p.stderr


def test_options_defaults_match_reference_constants(G):
    o = G.options()
    assert o.max_iter == 30 and abs(o.tol - 0.001) < 1e-15  # src/pr/pr.h:4-5
    assert np.float32(o.damping) == np.float32(0.85)        # include/common.h:18


def test_struct_layout_matches_header(G, tmp_path):
    """The ctypes mirrors have the C compiler's sizes and field offsets."""
    src = r"""
#include <stddef.h>
#include <stdio.h>
#include "gpr.h"
int main(void) {
  printf("%zu %zu %zu %zu %zu %zu %zu\n", sizeof(gpr_pr_opts), sizeof(gpr_pr_stats),
         sizeof(gpr_layout_opts), offsetof(gpr_pr_opts, variant),
         offsetof(gpr_pr_opts, timeout_s), offsetof(gpr_pr_stats, loop_ms),
         offsetof(gpr_pr_stats, gpu_launches));
  return 0;
}
"""
    c = tmp_path / "sz.c"
    c.write_text(src)
    exe = tmp_path / "sz"
    subprocess.run(["/usr/bin/gcc", "-std=c99", str(c), "-I", os.path.join(ROOT, "include"),
                    "-o", str(exe)], check=True)
    got = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True,
                                          check=True).stdout.split()]
    want = [C.sizeof(G.PrOptions), C.sizeof(G.PrStats), C.sizeof(G.LayoutOptions),
            G.PrOptions.variant.offset, G.PrOptions.timeout_s.offset, G.PrStats.loop_ms.offset,
            G.PrStats.gpu_launches.offset]
    assert got == want


@pytest.mark.skipif(has_gpu(), reason="checks the no-device path")
def test_no_device_reports_enodev(G):
    with pytest.raises(G.GprError) as e:
        G.Graph(np.array([0, 0], np.int32), np.array([], np.int32), np.array([0], np.int32))
    assert e.value.status == G.GPR_ENODEV
    with pytest.raises(G.GprError) as e:
        G.SpmvSolver(1, 0, np.array([0, 0], np.int32), np.array([], np.int32),
                     np.array([], np.float32), np.ones(1, np.float32), np.zeros(1, np.float32))
    assert e.value.status == G.GPR_ENODEV


def _strip_comments(src):
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def _function_body(src, signature):
    i = src.index("{", src.index(signature))
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j + 1]
    raise ValueError(signature)


def test_c_abi_never_exits_the_process():
    """Only the reference-shaped C++ drop-ins print and exit, as the reference
    does (gpr_dropin.cc, and read_graph in gpr_graph_io.cc); no other library
    source exits, aborts or traps, so a C-ABI caller always gets a status."""
    csrc = os.path.join(ROOT, "gardenia_ocl_b200", "csrc")
    checked = 0
    for name in sorted(os.listdir(csrc)):
        if not name.endswith((".cu", ".cc", ".cuh", ".h")) or name == "gpr_dropin.cc":
            continue
        src = _strip_comments(open(os.path.join(csrc, name)).read())
        if name == "gpr_graph_io.cc":
            src = src.replace(_function_body(src, "\nvoid read_graph("), "")
        assert not re.search(r"\b(exit|abort|quick_exit|_Exit|__trap)\s*\(", src), name
        checked += 1
    assert checked >= 15


@pytest.mark.parametrize("tol,max_iter", [(1e-3, 30), (0.0, 7), (1e-3, 0)])
def test_empty_graph_sweep_count_matches_oracle(G, O, tol, max_iter):
    """m = 0 needs no device: the no-allocation entry counts the empty sweeps
    the reference's loop counts (omp_base.cc:23-43), as the oracle does."""
    with np.errstate(divide="ignore"):
        _, ref_it, _ = O.pr_plain_f32(np.zeros(1, np.int32), np.zeros(0, np.int32),
                                      np.zeros(0, np.int32), tol=tol, max_iter=max_iter)
    st = G.pagerank_noalloc(0, 0, None, None, None, None, tol=tol, max_iter=max_iter)
    assert st.iterations == ref_it and st.residual == 0.0


def test_invalid_arguments_rejected_before_device(G):
    with pytest.raises(G.GprError) as e:
        G.Graph(np.array([0, 0], np.int32), np.array([], np.int32), np.array([0], np.int32),
                m=-1)
    assert e.value.status == G.GPR_EINVAL


@pytest.mark.gpu
def test_block_cache_reuses_and_releases(G):
    G.release_cached()
    p = C.c_void_p()
    assert G.lib().gpr_malloc(C.byref(p), 64 << 20) == 0
    first = p.value
    assert G.lib().gpr_free(p) == 0
    assert G.cached_bytes() >= 64 << 20
    q = C.c_void_p()
    assert G.lib().gpr_malloc(C.byref(q), (64 << 20) - 4096) == 0  # fits within 1/8
    assert q.value == first
    assert G.lib().gpr_free(q) == 0
    assert G.release_cached() >= 64 << 20 and G.cached_bytes() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("size", [1, 512, 513, 300000, 524288, 524289, (1 << 20) - 1, 1 << 20])
def test_small_blocks_are_kept_by_size_class(G, size):
    """A freed block comes back for the next request of its size class and holds what is
    written to it; release returns all of them."""
    G.release_cached()
    p, q, r = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert G.lib().gpr_malloc(C.byref(p), size) == 0
    assert G.lib().gpr_malloc(C.byref(q), size) == 0
    assert p.value != q.value
    first = q.value
    assert G.lib().gpr_free(q) == 0
    assert G.cached_bytes() >= size
    assert G.lib().gpr_malloc(C.byref(r), size) == 0
    assert r.value == first
    a = np.arange(size, dtype=np.int64).astype(np.uint8)
    b = np.zeros_like(a)
    for d, s in ((r, C.c_void_p(a.ctypes.data)), (C.c_void_p(b.ctypes.data), r)):
        assert G.lib().gpr_memcpy(d, s, size) == 0
    assert np.array_equal(a, b)
    assert G.lib().gpr_free(p) == 0 and G.lib().gpr_free(r) == 0
    assert G.release_cached() >= 2 * size and G.cached_bytes() == 0
