"""Threads per block of k_node and k_material: what a caller or the autotuner sets is
launched; the default gives way on small meshes."""
import ctypes
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), "/usr/local/cuda")
    d = tmp_path_factory.mktemp("blocks")
    src, so = str(d / "blocks.cpp"), str(d / "blocks.so")
    with open(src, "w") as f:
        f.write(f'#include "{ROOT}/lulesh.jl_gb300/csrc/lulesh_kernels.h"\n'
                'using namespace lulesh;\n'
                'extern "C" int node(int n, int b) { return threads_per_block(n, b, kNodeBlock); }\n'
                'extern "C" int mat(int n, int b) { return threads_per_block(n, b, kMatBlock); }\n'
                'extern "C" int same(const int* a, const int* b) {\n'
                '  Tuning x, y;\n'
                '  x.force = a[0]; x.node = a[1]; x.kin = a[2]; x.mat = a[3]; x.geo = a[4];\n'
                '  y.force = b[0]; y.node = b[1]; y.kin = b[2]; y.mat = b[3]; y.geo = b[4];\n'
                '  return same_launches(x, y);\n}\n')
    subprocess.run([os.environ.get("CXX") or shutil.which("g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
                    "-I", os.path.join(cuda, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("units", [1, 27, 512, 27000, 10 ** 6])
def test_set_sizes_are_launched(lib, units):
    assert [lib.node(units, b) for b in (128, 512)] == [128, 512]
    assert [lib.mat(units, b) for b in (64, 256)] == [64, 256]


@pytest.mark.parametrize("units", [1, 31, 512, 9261, 27000, 8 * 152 * 64, 8 * 152 * 128, 10 ** 6])
def test_default_sizes_follow_the_mesh(lib, units):
    for f, most in ((lib.node, 256), (lib.mat, 128)):
        b = f(units, most)
        assert b in (32, 64, 128, 256) and b <= most
        # the largest with eight blocks per SM, or a warp
        assert b == 32 or -(-units // b) >= 8 * 152
        assert b == most or -(-units // (2 * b)) < 8 * 152


def test_only_what_changes_a_launch_rebuilds_graphs(lib):
    """force_block, kin_block and geometry have no effect."""
    base = [128, 256, 128, 128, 0]
    for i, v in enumerate((64, 128, 64, 64, 1)):
        other = list(base)
        other[i] = v
        assert bool(lib.same((ctypes.c_int * 5)(*base), (ctypes.c_int * 5)(*other))) == (i in (0, 2, 4)), i
