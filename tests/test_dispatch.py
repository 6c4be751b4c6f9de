"""Which kernels a blob's steps launch, on both sides of each rule's line."""
import pytest

from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import kuhn_box
from test_cg_forms import fan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,solver,precision,kernel,shape", [
    # FP64: rows on chip by units up to 512 a block (77,824 rows), by the older form up to its shared memory, then neither
    ((6, 6, 6), "CG_nomass", "fp64", "cg_own_unit_kernel", (22, None, 16)),
    ((41, 42, 42), "CG_nomass", "fp64", "cg_own_unit_kernel", (152, 512, 511)),
    ((43, 42, 41), "CG_nomass", "fp64", "cg_own_kernel", (152, 1024, None)),
    ((76, 70, 70), "CG_nomass", "fp64", "cg_kernel", (152, 1024, 0)),
    # its consistent-mass form in one block while that holds a thread per component
    ((1, 4, 16), "CG", "fp64", "cg_own_unit_kernel", (1, 512, 170)),
    ((2, 2, 18), "CG", "fp64", "cg_own_unit_kernel", (11, None, 16)),
    # mixed CG_nomass: 128 rows a block while SMs are free, register blocks up to 512 rows, 100 MB of matrix, the rows that
    # fit on chip
    ((7, 3, 3), "CG_nomass", "mixed", "cg_mixed_sr_kernel", (1, 512, 128)),
    ((7, 4, 3), "CG_nomass", "mixed", "cg_mixed_sr_kernel", (2, 512, 80)),
    ((41, 42, 42), "CG_nomass", "mixed", "cg_mixed_sr_kernel", (152, 512, None)),
    ((43, 42, 41), "CG_nomass", "mixed", "cg_mixed_sr_kernel", (152, 1024, None)),
    ((52, 52, 52), "CG_nomass", "mixed", "cg_mixed_sr_kernel", (152, 1024, None)),
    ((55, 55, 55), "CG_nomass", "mixed", "cg_mixed_own_kernel", (152, 1024, None)),
    ((77, 75, 74), "CG_nomass", "mixed", "cg_mixed_kernel", (152, 1024, 0)),
    # mixed consistent mass: one block up to 512 rows, then 64 rows a block
    ((7, 7, 7), "CG", "mixed", "cg_mixed_own_kernel", (1, 1024, None)),
    ((8, 7, 7), "CG", "mixed", "cg_mixed_own_kernel", (9, 1024, 64)),
    ((2, 2, 2), "masslumped", "fp64", "none", (0, 0, 0)),
])
def test_cg_kernel(gpu, cells, solver, precision, kernel, shape):
    b = lib.Blob(kuhn_box(*cells, 5.0, seed=4), solver=solver, precision=precision)
    k = b.kernels()
    assert k["cg"] == kernel
    got = (k["cg_blocks"], k["cg_threads"], k["cg_rows"])
    assert all(want is None or g == want for g, want in zip(got, shape)), got


@pytest.mark.parametrize("cells,precision,kernel", [((11, 11, 13), "fp64", "element_split_kernel"),
                                                    ((12, 11, 13), "fp64", "element_kernel"),
                                                    ((11, 11, 13), "mixed", "element_mixed_kernel")])
def test_element_kernel(gpu, cells, precision, kernel):
    assert lib.Blob(kuhn_box(*cells, 3.0, seed=4), precision=precision).kernels()["element"] == kernel


@pytest.mark.parametrize("mesh,solver,precision,kernel", [
    (lambda: kuhn_box(15, 15, 17, 5.0, seed=4), "CG_nomass", "fp64", "assemble_kernel"),  # 144 slices of 32 rows
    (lambda: kuhn_box(16, 16, 16, 5.0, seed=4), "CG_nomass", "fp64", "assemble_rows_kernel"),  # 154
    (lambda: kuhn_box(1, 1, 1, 5.0, seed=4), "CG_nomass", "mixed", "assemble_rows_kernel"),
    (lambda: fan(62), "CG_nomass", "mixed", "assemble_rows_kernel"),  # rows of 64 blocks
    (lambda: fan(63), "CG_nomass", "mixed", "assemble_kernel"),
    (lambda: kuhn_box(1, 1, 1, 5.0, seed=4), "CG", "mixed", "none")])
def test_assembly_kernel(gpu, mesh, solver, precision, kernel):
    assert lib.Blob(mesh(), solver=solver, precision=precision).kernels()["assembly"] == kernel
