"""The launch sizes of csrc/cg_shapes.h, compiled for the host and read as the plans read them."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ffea_ci_demo_gb300", "csrc")
SRC = """
#include "cg_shapes.h"
extern "C" {
long long smem(int npb, int nhalo, int poly) { return (long long)ffea::sr_smem_bytes(npb, nhalo, poly); }
int recorded() { return ffea::CHEB_REC; }
int unit_grid(int n, int rows, int most) { return ffea::own_unit_grid(n, rows, most); }
int unit_sums() { return ffea::UNIT_SUM_BLOCKS; }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("shapes")
    (d / "shapes.cpp").write_text(SRC)
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "shapes.cpp"), "-o",
                    str(d / "libshapes.so")], check=True)
    lib = C.CDLL(str(d / "libshapes.so"))
    lib.smem.restype = C.c_longlong
    return lib


def test_lanczos_scratch_fits_the_smallest_blob(shapes):
    """The estimate of a blob's first solve keeps two doubles per recorded iteration in the block's dynamic shared
    memory; a one-element blob's rows (4, no halo) take 544 bytes."""
    for rows in range(1, 33):
        for halo in (0, 1, 40):
            for poly in (2, 4, 6, 8):
                got = shapes.smem(rows, halo, poly)
                assert got >= 16 * shapes.recorded()
                assert got >= 4 * 30 * rows + 16 * (rows + halo)  # and the rows' own fields
            assert shapes.smem(rows, halo, 0) == 4 * 24 * rows + 16 * (rows + halo)  # Jacobi alone records nothing


def test_unit_sums_hold_every_block(shapes):
    """The FP64 solve's sums over blocks hold 160 partials: no device's grid exceeds that, and no row is left out."""
    for most in (1, 80, 152, 160, 161, 208, 1000):
        for rows in (16, 64, 512):
            for n in (1, rows, rows + 1, 2197, 77824, 200000):
                g = shapes.unit_grid(n, rows, most)
                assert 1 <= g <= min(most, shapes.unit_sums())
                assert g == most or g == shapes.unit_sums() or g * rows >= n
