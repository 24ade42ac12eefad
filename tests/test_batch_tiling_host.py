"""The numbers of the batched sweeps' tile shapes, which programs keep from one
run to the next (cfd_batch_autotune's choice, cfd_batch_set_tiling's argument):
shape 0 takes 4 lines a tile along x and 32 along y and z, shape 1 16 along y
and z and 8 along x."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("tiling") / "libtiling.so"
    subprocess.run([nvcc, "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "cfd_inwsl_b200" / "csrc"), str(ROOT / "tests" / "tiling_host.cu"), "-o", str(out)],
                   check=True, capture_output=True)
    f = C.CDLL(str(out)).h_batch_tiles
    f.restype = C.c_longlong
    return f


@pytest.mark.parametrize("shape,lines", [(0, (4, 32, 32)), (1, (8, 16, 16))])
def test_shape_numbers(tiles, shape, lines):
    n = 96
    for dim in (2, 3):
        nz = n if dim == 3 else 1
        for ax in range(dim):
            want = n // lines[ax] * nz * 2  # two segments a line
            assert tiles(dim + 2, ax, n, n, nz, n // 2, 0, shape) == want
