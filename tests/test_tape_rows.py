"""The adjoint's tapes hold up to 90 rows of one entry per element, so from 288^3
elements on their entries lie past 2^31: the index every kernel forms them with
is compiled for the host and compared with exact integers, and no kernel source
may form one with a 32-bit product."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "lulesh.jl_gb300", "csrc")
ROWS = 90  # DevDomain::tapeKin, the tape with the most


@pytest.fixture(scope="module")
def row(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), "/usr/local/cuda")
    d = tmp_path_factory.mktemp("rows")
    src, so = str(d / "rows.cpp"), str(d / "rows.so")
    with open(src, "w") as f:
        f.write(f'#include "{CSRC}/lulesh_internal.h"\n'
                'extern "C" unsigned long long row(int slot, int E, int e) { return lulesh::row(slot, E, e); }\n')
    subprocess.run([os.environ.get("CXX") or shutil.which("g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
                    "-I", os.path.join(cuda, "include"), src, "-o", so], check=True)
    f = ctypes.CDLL(so).row
    f.restype = ctypes.c_ulonglong
    return f


@pytest.mark.parametrize("nx", [1, 287, 288, 448, 640])
def test_rows_past_31_bits(row, nx):
    E = nx ** 3
    for slot in (0, 1, 23, 65, ROWS - 1):
        for e in (0, E // 2, E - 1):
            assert row(slot, E, e) == slot * E + e, (slot, e)


def test_only_the_connectivity_is_indexed_in_32_bits():
    """8 rows (connectivity, corner forces) stay below 2^31 by the limit on nx."""
    assert 8 * 640 ** 3 < 2 ** 31 < ROWS * 288 ** 3
    for name in ("lulesh_kernels.cu", "lulesh_adjoint_kernels.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            for m in re.finditer(r"(\w+)\[[^\[\]]*\*\s*(?:d\.|a\.)?E\b[^\[\]]*\]", f.read()):
                assert m.group(1) in ("nodelist", "out"), (name, m.group(0))
