"""The tiles of the resident Jacobi sweeps (csrc/jacobi_tiles.h, host arithmetic, compiled here with the
host compiler): they cover the grid, fit the shared memory, and never outnumber the CTAs that a
cooperative launch may have, whatever the device has left of it."""
import ctypes
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = """
#include "jacobi_tiles.h"
extern "C" int tiles(int real, int n, int nz, int sms, int resident, int* out) {
    shg::ResidentTiles t;
    if (!shg::resident_tiles((size_t)real, n, nz, sms, resident, &t)) return 0;
    out[0] = t.ytiles; out[1] = t.tz; out[2] = t.ztiles;
    return 1;
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cpp").write_text(SRC)
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "cushg_b200", "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    lib = ctypes.CDLL(str(d / "t.so"))

    def call(real, n, nz, sms, resident):
        out = (ctypes.c_int * 3)()
        return tuple(out) if lib.tiles(real, n, nz, sms, resident, out) else None

    return call


def test_no_device_or_too_few_multiprocessors_fits_nothing(tiles):
    assert tiles(8, 32, 4, 0, 0) is None
    assert tiles(4, 256, 4, 0, 148) is None
    assert tiles(4, 256, 20, 40, 40) is None      # 64 tiles along y alone
    assert tiles(4, 256, 20, 148, 40) is None     # a partition of the device
    assert tiles(8, 128, 100, 148, 0) is None     # the kernel does not fit a multiprocessor
    assert tiles(8, 96, 20, 148, 148) is None
    assert tiles(8, 128, 200, 148, 148) == (16, 23, 9)


@pytest.mark.parametrize("real", [4, 8])
@pytest.mark.parametrize("n", [32, 64, 128, 256])
def test_tiles_cover_the_grid_and_fit(tiles, real, n):
    for sms in (1, 7, 64, 100, 132, 148, 160):
        for nz in range(1, 500):
            t = tiles(real, n, nz, sms, sms)
            if t is None:
                continue
            ytiles, tz, ztiles = t
            assert ytiles * (1024 // n) == n
            assert (ztiles - 1) * tz < nz <= ztiles * tz
            assert real * 1024 * tz <= 208 * 1024 and ytiles * ztiles <= sms
