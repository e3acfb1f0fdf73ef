"""The block count of the fused half iterations (falm_b200/csrc/pc_tile.cuh, plain
host C++ compiled here with g++): every block has a slot of the reduction workspace."""
import ctypes
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAX_BLOCKS = 1 << 16   # RedWork::maxBlocks

SHIM = """
#include "pc_tile.cuh"
using namespace fb;
#define FORWARD(S, T)                                                                                                    \\
    extern "C" int chunk_##S(int nx, int ny, int nz, int sms, int mb) { return pc_chunk<T>(nx, ny, nz, sms, mb); }        \\
    extern "C" long long tiles_##S(int nx, int ny) { return (long long)PCTile<T>::tiles_x(nx) * PCTile<T>::tiles_y(ny); } \\
    extern "C" int kmax_##S() { return PCTile<T>::KMAX; }
FORWARD(fp64, double)
FORWARD(fp32, float)
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("pc_tile")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "falm_b200", "csrc"), str(d / "shim.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    for t in ("fp64", "fp32"):
        getattr(lib, "tiles_" + t).restype = ctypes.c_longlong
    return lib


def shapes():
    rng = random.Random(3)
    # wide shallow grids whose tiles alone exceed the workspace, then grids at its edge, then any
    yield from [(8192, 8192, 4), (16384, 4096, 1), (7700, 7700, 3), (20000, 20000, 1), (1 << 20, 64, 1)]
    yield from [(14344, 4104, 1), (14344, 4104, 96), (14344, 4104, 97), (7176, 4104, 200), (56 * 256 + 8, 24 * 256 + 8, 2)]
    for _ in range(300):
        yield tuple(int(10 ** rng.uniform(0, 4.3)) for _ in range(2)) + (int(10 ** rng.uniform(0, 3.3)),)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sms", [148, 132, 1])
def test_every_block_has_a_workspace_slot(rule, precision, sms):
    """A chunk is at most KMAX planes long and gives at most MAX_BLOCKS blocks; none (0)
    is returned exactly where the longest chunk already gives more."""
    kmax = getattr(rule, "kmax_" + precision)()
    refused = 0
    for nx, ny, nz in shapes():
        kc = getattr(rule, "chunk_" + precision)(nx, ny, nz, sms, MAX_BLOCKS)
        tiles = getattr(rule, "tiles_" + precision)(nx, ny)
        fewest = tiles * -(-nz // min(nz, kmax))
        assert (kc == 0) == (fewest > MAX_BLOCKS), (nx, ny, nz, kc)
        refused += kc == 0
        if kc:
            assert 1 <= kc <= min(nz, kmax) and tiles * -(-nz // kc) <= MAX_BLOCKS, (nx, ny, nz, kc)
    assert refused > 4
