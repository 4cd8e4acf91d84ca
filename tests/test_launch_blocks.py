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
                'extern "C" int mat(int n, int b) { return threads_per_block(n, b, kMatBlock); }\n')
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
