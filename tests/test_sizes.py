"""Size rules of the engine (csrc/sizes.hpp) on the host, over all shapes that
lat_create accepts (6 (nx/2+1) ny nz below 2^31): long thin boxes and wide ones."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
BINS = 2048
SHAPES = [(2, 2, 2), (3, 2, 5), (64, 64, 64), (512, 512, 512), (1024, 768, 512), (4096, 2, 2), (4097, 3, 2),
          (16384, 16, 16), (65536, 8, 4), (131072, 2, 2), (2, 131072, 2), (2, 2, 131072), (92682, 4, 4),
          (50000, 50000, 2), (2, 10000, 17000), (178956900, 2, 2), (2, 44739242, 2), (2, 2, 44739242)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("sizes") / "libsizes.so"
    subprocess.run(["g++", "-O1", "-std=gnu++17", "-shared", "-fPIC", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-o", str(so), str(HERE / "sizes.cpp")], check=True)
    lib = C.CDLL(str(so))
    lib.bin_table.restype = C.c_longlong
    return lib


@pytest.mark.parametrize("shape", SHAPES)
def test_shell_tables(lib, shape):
    """The tables hold every |n|^2 of the lattice below 2048^2, the end of the
    last shell, and no more than that."""
    n = lib.bin_table(*shape)
    top = sum((s // 2) ** 2 for s in shape)
    assert n == min(top + 1, BINS ** 2)
    assert 24 * n <= 101 * 2 ** 20  # weights and counts


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("shape", SHAPES + [(2, 262140, 2), (2, 262141, 2), (64, 262200, 3), (2, 524280, 4),
                                            (2, 2, 4194240), (2, 4, 4194300)])
def test_default_stencil_tile(lib, shape, fp64):
    """The untuned stencil pass of every lattice has a grid: rows of blocks along y and chunks along z
    are at most 65535 up to 524280 rows (8 a block, as far as an untuned pass ever went; 16 beyond)."""
    nx, ny, nz = shape
    out = (C.c_int * 3)()
    lib.fd_tile(nx, ny, nz, fp64, 152, out)
    ty, zc, fits = out
    assert 1 <= zc <= nz and ty == (4 if ny <= 4 * 65535 else 8 if ny <= 8 * 65535 else 16)
    assert -(-nz // zc) <= 65535
    assert bool(fits) == (-(-ny // ty) <= 65535)
