"""Launch shapes of the marching passes (csrc/launch_shapes.h): every chunk count fits a
launch's extents, and the choices on the grids that the rules were measured on."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("shapes")
    src = d / "shapes.cpp"
    src.write_text('#include "launch_shapes.h"\n'
                   'extern "C" int rows(long y, long s, int t, int w, long n) { return crp::march_rows(y, s, t, w, n); }\n'
                   'extern "C" int planes(long z, long b, int n) { return crp::march3_planes(z, b, n); }\n')
    out = d / "libshapes.so"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "cuda-rp_b200", "csrc"),
                    "-o", str(out), str(src)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.rows.argtypes = [ctypes.c_long, ctypes.c_long, ctypes.c_int, ctypes.c_int, ctypes.c_long]
    lib.planes.argtypes = [ctypes.c_long, ctypes.c_long, ctypes.c_int]
    return lib


def test_rows(lib):
    # 64 columns per strip, 4 warps per block, 4 blocks on each of 148 SMs.
    for x, y, tuned, want in ((600, 701, 8, 3), (1001, 1531, 8, 4), (1024, 2048, 8, 4), (256, 512, 8, 1),
                              (256, 512, 4, 1), (64, 20000, 8, 3), (64, 20000, 4, 2), (64, 20000, 16, 5)):
        assert lib.rows(y, (x + 63) // 64, tuned, 4, 4 * 148) == want, (x, y, tuned)


def test_planes(lib):
    for (x, y, z), want in (((256, 256, 256), 16), ((384, 384, 384), 16), ((141, 125, 133), 8), ((12, 12, 12), 2)):
        assert lib.planes(z, (x + 63) // 64 * ((y + 7) // 8), 148) == want, (x, y, z)


@pytest.mark.parametrize("z", [65535 * 2, 65535 * 16, 65535 * 16 + 1, 65535 * 32, 2**24 - 1])
@pytest.mark.parametrize("blocks", [1, 64, 10**6])
def test_chunks_of_long_grids_fit_a_launch(lib, z, blocks):
    planes = lib.planes(z, blocks, 148)
    assert planes >= 2 and -(-z // planes) <= 65535
