"""The CG solves at the ends of their ranges: tiny forces, the smallest blobs."""
import numpy as np
import pytest

from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import apply_shear, kuhn_box


# |f|^2 of about 1e-25 and 1e-27: the tolerance 1e-20 |f|^2 (1e-45, 1e-47) is at and below FP32's smallest number, |r|^2
# rounds to zero first and is less than it in FP64. Viscosity (and density) keep the diagonal below 1, so that r.z and p.q
# outlast |r|^2. The mixed path's bound against FP64 (velocities: the moves are below the positions' rounding).
@pytest.mark.gpu
@pytest.mark.parametrize("solver,kernel", [("CG_nomass", "cg_mixed_sr_kernel"), ("CG", "cg_mixed_own_kernel")])
@pytest.mark.parametrize("scale", [1e-10, 1e-11])
def test_mixed_solve_of_a_tiny_force_converges(gpu, solver, kernel, scale):
    m = kuhn_box(3, 3, 3, 5.0, seed=4)
    m.material = m.material.copy()
    m.material[:, 3:5] *= scale
    m.material[:, 1:3] *= 1e-3 if solver == "CG_nomass" else 1e-6
    m.material[:, 0] *= 1.0 if solver == "CG_nomass" else 1e-6
    v = {}
    for prec in ("fp64", "mixed"):
        b = lib.Blob(m, solver=solver, precision=prec, dt=1e-16, kT=0.0, calc_noise=0)
        b.set_state(pos=apply_shear(m, 1e-6) * (m.scale / 1.7e-10))
        b.update(1)
        v[prec] = b.vel()
    assert b.cg_kernel() == kernel
    assert 0 < (b.rhs() ** 2).sum() < 1e-24
    assert np.abs(v["mixed"] - v["fp64"]).max() < 1e-5 * np.abs(v["fp64"]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["CG_nomass", "CG"])
def test_one_element_blob(gpu, solver):
    """A single tetrahedron: four rows, its first solve's Lanczos record and the polynomial's solves after it."""
    from test_mixed_elements import one_tet

    m = one_tet()
    kw = dict(solver=solver, dt=1e-14, kT=4.11e-21, calc_noise=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    out = {}
    for prec in ("fp64", "mixed"):
        b = lib.Blob(m, precision=prec, **kw)
        b.set_state(pos=p0)
        b.update(4)
        out[prec] = b.pos()
    assert np.abs(out["mixed"] - out["fp64"]).max() < 1e-5 * np.abs(out["fp64"] - p0).max()


# the CG kernels of the largest mixed blobs, each row count leaving the last block and the last slice short: rows on chip
# with a matrix above 100 MB (and the consistent-mass solve by the same kernel), and the grid-strided kernel beyond its
# rows, both forms. One step against the FP64 path, the mixed path's bound
@pytest.mark.gpu
@pytest.mark.parametrize("cells,solver,kernel", [((55, 54, 53), "CG_nomass", "cg_mixed_own_kernel"),
                                                 ((55, 54, 53), "CG", "cg_mixed_own_kernel"),
                                                 ((77, 75, 74), "CG_nomass", "cg_mixed_kernel"),
                                                 ((77, 75, 74), "CG", "cg_mixed_kernel")])
def test_largest_mixed_blobs(gpu, cells, solver, kernel):
    m = kuhn_box(*cells, 5.0, seed=4)
    kw = dict(solver=solver, dt=1e-13 if solver == "CG_nomass" else 1e-14, kT=4.11e-21, calc_noise=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    out = {}
    for prec in ("fp64", "mixed"):
        b = lib.Blob(m, precision=prec, **kw)
        b.set_state(pos=p0)
        b.update(1)
        out[prec] = b.pos()
        if prec == "mixed":
            assert b.cg_kernel() == kernel
        b.close()
    assert np.abs(out["mixed"] - out["fp64"]).max() < 1e-5 * np.abs(out["fp64"] - p0).max()


@pytest.mark.gpu
def test_batch_waits_outlast_another_blobs_solve(gpu):
    """Two blobs that need 125 of the 152 blocks each: the second's first blocks wait for the rest through the whole of
    the first's solve, which here never converges (a tolerance of zero) and takes about three seconds, longer than a
    wait without progress may take. The step ends with the iteration cap, not with a timeout."""
    m = kuhn_box(39, 39, 39, 5.0, seed=4)
    bt = lib.Batch([m, m], dt=1e-13, kT=4.11e-21, epsilon=0.0, max_iterations_cg=250_000)
    with pytest.raises(lib.FFEAError) as e:
        bt.update(1)
    assert e.value.code == lib.ECGMAXIT
    assert list(bt.cg_iterations()[0]) == [250_000, 250_000]


# the FP64 consistent-mass solve on both sides of one block's 170 rows, against the oracle's CG
@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(1, 4, 16), (2, 2, 18)])
def test_consistent_mass_one_block_edge(gpu, oracle_built, cells):
    import pyoracle

    m = kuhn_box(*cells, 5.0, seed=4)
    kw = dict(solver="CG", dt=1e-14, kT=4.11e-21, calc_noise=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    b, o = lib.Blob(m, **kw), pyoracle.OracleBlob(m, threads=1, fast=True, **kw)
    b.set_state(pos=p0)
    o.set_pos(p0)
    b.update(2)
    assert o.step(2) == 0
    moved = np.abs(o.pos() - p0).max()
    assert np.abs(b.pos() - o.pos()).max() < 1e-8 * moved + 1e-15 * np.abs(p0).max()
