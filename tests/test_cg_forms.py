"""The mixed CG_nomass solve (cg_mixed_sr_kernel) at the edges of its launch forms, against the FP64 path."""
import numpy as np
import pytest

from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import apply_shear, kuhn_box


# rows per block of the single-reduction CG at the edges of its forms: one block (8 and 128 rows), two blocks,
# a row count that leaves the last block short, the register form's last lanes-per-row steps, and (42^3 cells, 523
# rows a block) the form without register blocks; the shuffled numbering gives every block a halo of most of the mesh
@pytest.mark.gpu
@pytest.mark.parametrize("cells,shuffle", [((1, 1, 1), False), ((7, 3, 3), False), ((7, 4, 4), False),
                                           ((33, 9, 7), True), ((20, 20, 20), True), ((30, 29, 31), False),
                                           ((42, 42, 42), False)])
def test_single_reduction_cg_forms(cells, shuffle):
    m = kuhn_box(*cells, 5.0, seed=4)
    if shuffle:  # vertices renumbered at random: the same blob in another node order
        rng = np.random.default_rng(9)
        new = np.concatenate([rng.permutation(m.n_linear), np.arange(m.n_linear, m.n_nodes)])
        pos = np.empty_like(m.pos)
        pos[new] = m.pos
        m.pos, m.tets = pos, new[m.tets].astype(np.int32)
    kw = dict(solver="CG_nomass", dt=1e-13, kT=4.11e-21, calc_noise=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    out = {}
    for prec, extra in (("fp64", {}), ("mixed", {}), ("mixed", {"cg_smem_blocks": -1})):
        b = lib.Blob(m, precision=prec, **kw, **extra)
        b.set_state(pos=p0)
        b.update(3)  # Jacobi, the polynomial's trial, the polynomial
        out[prec, bool(extra)] = b.pos()
        if prec == "mixed":
            assert b.cg_kernel() == "cg_mixed_sr_kernel"
    move = np.abs(out["fp64", False] - p0).max()
    assert np.abs(out["mixed", False] - out["fp64", False]).max() < 1e-5 * move  # the mixed path's bound
    assert np.array_equal(out["mixed", False], out["mixed", True])  # where the matrix is read from does not matter
