"""The C ABI library (no GPU): it builds for sm_100a, loads, and exports every
entry point declared in include/qpgpu.h."""
import ctypes as C
import os
import subprocess

import pytest


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    if not os.path.exists(qpgpu.LIB_PATH):
        qpgpu.build()
    return qpgpu


def test_library_exports_every_declared_symbol(qp):
    L = qp.lib()
    syms = qp.exported_symbols()
    assert len(syms) > 50
    missing = [s for s in syms if not hasattr(L, s)]
    assert not missing, missing


def test_library_has_no_cuda_runtime_dependency(qp):
    """cudart is linked statically, so the library loads wherever the driver is."""
    out = subprocess.run(["ldd", qp.LIB_PATH], capture_output=True, text=True).stdout
    assert "libcudart" not in out


def test_errors_are_reported_not_crashed(qp):
    """A bad grid is rejected with a message before any device call."""
    L = qp.lib()
    with pytest.raises(qp.QPError, match="grid exponents"):
        qp.Context(2, 2, 2, [[-1, 1], [-1, 1], [0, 1]])
    assert b"grid exponents" in L.qp_ctx_last_error(None)


def test_oracle_is_not_linked_by_the_product(qp):
    out = subprocess.run(["ldd", qp.LIB_PATH], capture_output=True, text=True).stdout
    assert "oracle" not in out
    nm = subprocess.run(["nm", "-D", qp.LIB_PATH], capture_output=True, text=True).stdout
    assert "oq_" not in nm


# (C struct in include/qpgpu.h, ctypes mirror in qpgpu) pairs of the boundary
STRUCTS = [("qp_grid_desc", "_GridDesc"), ("qp_species_desc", "_SpeciesDesc"),
           ("qp_beam_desc", "_BeamDesc"), ("qp_sim_desc", "_SimDesc"),
           ("qp_step_stats", "StepStats"), ("qp_scan_desc", "_ScanDesc"),
           ("qp_scan_stats", "ScanStats"), ("qp_nn_train_desc", "_TrainDesc"),
           ("qp_nn_train_stats", "TrainStats")]


def test_descriptor_layouts_match_the_header(qp, tmp_path):
    """Every descriptor's size and field offsets, as the C compiler lays them
    out from include/qpgpu.h, equal the ctypes mirror's (a drifted field would
    pass wrong values across the boundary without any error)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lines = ["#include <stdio.h>", "#include <stddef.h>", '#include "qpgpu.h"', "int main(void) {"]
    for cname, pyname in STRUCTS:
        lines.append(f'  printf("{pyname} size %zu\\n", sizeof({cname}));')
        for fname, _ in getattr(qp, pyname)._fields_:
            lines.append(f'  printf("{pyname} {fname} %zu\\n", offsetof({cname}, {fname}));')
    lines += ["  return 0;", "}"]
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines) + "\n")
    exe = tmp_path / "layout"
    subprocess.run(["gcc", "-std=c99", "-I", os.path.join(root, "include"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = {}
    for line in out.splitlines():
        name, field, val = line.split()
        got[(name, field)] = int(val)
    for _, pyname in STRUCTS:
        st = getattr(qp, pyname)
        assert got[(pyname, "size")] == C.sizeof(st), pyname
        for fname, _ in st._fields_:
            assert got[(pyname, fname)] == getattr(st, fname).offset, (pyname, fname)


def test_component_values_may_be_one_number(qp):
    """Field2d.mult with component lists takes a sequence of values or one
    number; what reaches the C call is one value per component."""
    import types

    import numpy as np

    seen = []

    def comp(h, a1, dim, dim1, value, n):
        seen.append((list(dim), list(dim1), list(value), n))
        return 0

    f = qp.Field2d.__new__(qp.Field2d)
    f.h = 1
    f.ctx = types.SimpleNamespace(_L=types.SimpleNamespace(qp_field2d_mult_comp=comp),
                                  _check=lambda rc: rc)
    for value, want in [(2.0, [2.0]), (3, [3.0]), (np.float32(0.5), [0.5]), (np.array(4.0), [4.0]),
                        ([1.5], [1.5]), (np.array([2.5]), [2.5])]:
        f.mult(f, value, dim=[1], dim1=[2])
        assert seen[-1] == ([1], [2], want, 1)
    f.mult(f, 2.0, dim=[1, 3], dim1=(2, 1))
    assert seen[-1] == ([1, 3], [2, 1], [2.0, 2.0], 2)
    f.mult(f, [2.0, 3.0], dim=np.array([1, 2]), dim1=[2, 1])
    assert seen[-1] == ([1, 2], [2, 1], [2.0, 3.0], 2)


def test_layout_conversion_counts_in_64_bits(tmp_path):
    """A beam may have more than 2^31 particles: the conversion's extents and
    indices, compiled for the host from the kernels' header."""
    src = tmp_path / "pack.cu"
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "quickpic-opensource_b200", "csrc")
    src.write_text("""
#include "qp_misc.cuh"
#include <cstdio>
int main() {
  qp::PackJob j{};
  const long long np = 3000000001LL;
  j.dim = 7;
  j.n0 = np;
  j.n1 = j.valid1 = 1;
  j.stride = 1;
  int bad = j.n0 != np;
  for (long long a : {0LL, 1LL, (1LL << 31) - 1, 1LL << 31, np - 1})
    for (int k = 0; k < 7; ++k) {
      int c = -1;
      long long at = -1;
      bad += !qp::pack_at(j, k + 7 * a, &c, &at) || c != k || at != a;
    }
  j.dim = 3;  // and slow indices past 2^31
  j.n0 = 18;
  j.n1 = j.valid1 = np;
  j.pitch = 20;
  int c;
  long long at;
  bad += !qp::pack_at(j, 2 + 3 * (5 + 18 * (np - 1)), &c, &at) || c != 2 || at != 20 * (np - 1) + 5;
  bad += qp::pack_at(j, 54 * np, &c, &at);
  return bad;
}
""")
    exe = tmp_path / "pack"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--expt-relaxed-constexpr", "-I", csrc, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
