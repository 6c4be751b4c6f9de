"""The CG kernels at the edges of their launch forms: the mixed CG_nomass solve (cg_mixed_sr_kernel) against the FP64
path, the FP64 solve against the oracle."""
import numpy as np
import pytest

import pyoracle
from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import MID_EDGES, Mesh, apply_shear, kuhn_box


def renumbered(m, shuffle):
    """The same blob with its vertices numbered at random (a block's halo is then most of the mesh)."""
    if shuffle:
        new = np.concatenate([np.random.default_rng(9).permutation(m.n_linear), np.arange(m.n_linear, m.n_nodes)])
        pos = np.empty_like(m.pos)
        pos[new] = m.pos
        m.pos, m.tets = pos, new[m.tets].astype(np.int32)
    return m


# rows per block of the single-reduction CG at the edges of its forms: one block (8 and 128 rows), two blocks,
# a row count that leaves the last block short, the register form's last lanes-per-row steps, and (42^3 cells, 523
# rows a block) the form without register blocks; the shuffled numbering gives every block a halo of most of the mesh
@pytest.mark.gpu
@pytest.mark.parametrize("cells,shuffle", [((1, 1, 1), False), ((7, 3, 3), False), ((7, 4, 4), False),
                                           ((33, 9, 7), True), ((20, 20, 20), True), ((30, 29, 31), False),
                                           ((42, 42, 42), False)])
def test_single_reduction_cg_forms(cells, shuffle):
    m = renumbered(kuhn_box(*cells, 5.0, seed=4), shuffle)
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


# the FP64 solve (cg_own_unit_kernel) at the edges of its forms, against the oracle's CG: one block, several, a halo
# of most of the mesh, one unit per component up to 170 rows a block, per row from there, and (44^3 cells, 600 rows a
# block) beyond the kernel
@pytest.mark.gpu
@pytest.mark.parametrize("cells,solver,shuffle", [((1, 1, 1), "CG", False), ((3, 3, 3), "CG", False),
                                                  ((4, 3, 3), "CG_nomass", False), ((12, 12, 12), "CG_nomass", True),
                                                  ((28, 28, 29), "CG", False), ((29, 28, 29), "CG_nomass", False),
                                                  ((31, 31, 31), "CG", True), ((31, 31, 31), "CG_nomass", False),
                                                  ((44, 44, 44), "CG", False)])
def test_fp64_cg_forms(cells, solver, shuffle):
    m = renumbered(kuhn_box(*cells, 5.0, seed=4), shuffle)
    kw = dict(solver=solver, dt=1e-13 if solver == "CG_nomass" else 1e-14, kT=4.11e-21, calc_noise=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    b = lib.Blob(m, **kw)
    o = pyoracle.OracleBlob(m, threads=1, fast=True, **kw)
    b.set_state(pos=p0)
    o.set_pos(p0)
    b.update(2)
    assert o.step(2) == 0
    assert b.cg_kernel() == "cg_own_kernel"
    moved = np.abs(o.pos() - p0).max()
    assert np.abs(b.pos() - o.pos()).max() < 1e-8 * moved + 1e-15 * np.abs(p0).max()  # and the positions' rounding
    h = b.cg_history()
    assert len(h) == b.cg_iterations()[0] and h[-1] < 1e-20 <= h[-2]  # the stopping test's own quantity


# the FP64 element phase's two forms (four lanes to an element up to 9,728 elements) at their edges, against the
# oracle: forces, volumes and positions bit for bit, the inertial solvers' viscous term and the noise included
@pytest.mark.gpu
@pytest.mark.parametrize("cells,solver,noise", [((1, 1, 1), "masslumped", 1), ((3, 5, 7), "masslumped", 0),
                                                ((3, 5, 7), "CG_nomass", 1), ((11, 11, 13), "masslumped", 1),
                                                ((12, 11, 13), "masslumped", 1)])
def test_fp64_element_forms(cells, solver, noise):
    m = kuhn_box(*cells, 3.0, seed=4)
    kw = dict(solver=solver, dt=1e-14, kT=4.11e-21, calc_noise=noise)
    p0 = apply_shear(m, 0.01, seed=5) * (m.scale / 1.7e-10)
    b, o = lib.Blob(m, **kw), pyoracle.OracleBlob(m, threads=1, **kw)
    b.set_state(pos=p0)
    o.set_pos(p0)
    n = 1 if solver == "CG_nomass" else 3
    b.update(n)
    assert o.step(n) == 0
    assert np.array_equal(b.rhs(), o.rhs()) and np.array_equal(b.rng_state(), o.rng_state())
    if solver == "masslumped":
        assert np.array_equal(b.pos(), o.pos()) and np.array_equal(b.vel(), o.vel())


# the batch's solve on chip at its edges: blobs of one block and of many, more tasks than SMs, and (610 blobs, four
# times the SMs and two) beyond it; each blob as the single mixed blob from the same state, and the same bits again
@pytest.mark.gpu
@pytest.mark.parametrize("cells", [[(7, 7, 7), (8, 7, 7)], [(12, 12, 12), (2, 2, 2), (20, 19, 21), (1, 1, 1)],
                                   [(3, 3, 3)] * 200 + [(9, 9, 9)], [(33, 33, 33), (31, 30, 32)], [(2, 2, 1)] * 610])
def test_batch_solve_forms(cells):
    box = {c: kuhn_box(*c, 5.0, seed=4) for c in set(cells)}
    meshes = [box[c] for c in cells]
    kw = dict(dt=1e-13, kT=4.11e-21, calc_noise=1)
    x0 = [apply_shear(m, 0.001) * (m.scale / 1.7e-10) for m in meshes]
    runs = []
    for _ in range(2):
        bt = lib.Batch(meshes, **kw)
        bt.set_positions(np.concatenate(x0))
        bt.update(4)
        runs.append(bt.positions())
    assert np.array_equal(*runs)
    for b in sorted({0, 1, len(meshes) // 2, len(meshes) - 1}):
        s = lib.Blob(meshes[b], precision="mixed", rng_state=lib.Batch(meshes[:b + 1], **kw).rng_state(b), **kw)
        s.set_state(pos=x0[b])
        s.update(4)
        assert np.abs(bt.pos(b) - s.pos()).max() < 1e-5 * np.abs(s.pos() - x0[b]).max(), b
        assert np.array_equal(bt.rng_state(b), s.rng_state()), b


# the FP64 assembly by rows (152 slices of 32 rows and more) beside the assembly by slots, against the oracle's matrix:
# the last size by slots and the first by rows, pinned vertices and a Stokes drag on the diagonal
@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(15, 15, 17), (16, 16, 16), (17, 17, 15)])
def test_fp64_assembly_forms(cells):
    m = kuhn_box(*cells, 5.0, seed=4)
    m.pinned = np.nonzero(m.pos[:m.n_linear, 0] == 0.0)[0].astype(np.int32)
    kw = dict(solver="CG_nomass", dt=1e-13, kT=4.11e-21, calc_noise=1, calc_stokes=1)
    p0 = apply_shear(m, 0.001) * (m.scale / 1.7e-10)
    p0[m.pinned] = m.pos[m.pinned] * (m.scale / 1.7e-10)
    b, o = lib.Blob(m, **kw), pyoracle.OracleBlob(m, threads=1, **kw)
    b.set_state(pos=p0)
    o.set_pos(p0)
    b.update(1)
    assert o.step(1) == 0
    g, c = b.pattern(), o.csr()
    assert np.array_equal(g["key"], c["key"]) and np.array_equal(g["col"], c["col"])
    assert np.array_equal(g["val"], c["val"])


def fan(n, r=5.0, h=5.0):
    """n elements around one edge, whose two vertices have rows of n + 2 blocks (pinned vertices have none)."""
    th = 2 * np.pi * np.arange(n) / n
    lin = np.vstack([[[0, 0, 0], [0, 0, h]], np.stack([r * np.cos(th), r * np.sin(th), np.full(n, 0.5 * h)], 1)])
    i = np.arange(n)
    t4 = np.stack([0 * i, 2 + i, 2 + (i + 1) % n, 1 + 0 * i], 1)
    mid, tets = {}, []
    for t in t4:
        tets.append(list(t) + [mid.setdefault(tuple(sorted((t[a], t[b]))), n + 2 + len(mid)) for a, b in MID_EDGES])
    pos = np.vstack([lin] + [0.5 * (lin[a] + lin[b])[None] for a, b in mid])
    b = kuhn_box(1, 1, 1, h)
    return Mesh(pos=pos, tets=np.array(tets, np.int32), material=np.tile(b.material[:1], (n, 1)),
                stokes_radius=np.full(len(pos), 1.0), scale=b.scale, n_linear=n + 2)


# the FP32 assembly: a ragged slice, whole slices and some rows more, three pins, and rows of 64 blocks (the widest by
# rows) and 65 (by slots). An FP32 gradient is off by some 16 roundings, times 1 / sin of the narrowest angle through
# the determinant; an entry has two gradients, a volume and two dozen additions: 128 roundings of the row's largest
@pytest.mark.gpu
@pytest.mark.parametrize("mesh,angle", [(lambda: kuhn_box(1, 1, 1, 5.0, seed=4), 0.5),
                                        (lambda: kuhn_box(7, 1, 1, 5.0, seed=4), 0.5),
                                        (lambda: kuhn_box(10, 2, 1, 5.0, seed=4), 0.5),
                                        (lambda: kuhn_box(9, 9, 9, 5.0, seed=4), 0.5),
                                        (lambda: fan(65), 2 * np.pi / 65), (lambda: fan(66), 2 * np.pi / 66)])
def test_mixed_assembly_forms(mesh, angle):
    m = mesh()
    m.pinned = np.arange(2, 5, dtype=np.int32)
    kw = dict(solver="CG_nomass", dt=1e-16, kT=4.11e-21, calc_noise=0, calc_stokes=1)
    b, o = lib.Blob(m, precision="mixed", **kw), pyoracle.OracleBlob(m, threads=1, **kw)
    b.update(1)
    assert o.step(1) == 0
    g, c = b.pattern(), o.csr()
    assert np.array_equal(g["key"], c["key"]) and np.array_equal(g["col"], c["col"])
    scale = np.maximum.reduceat(np.abs(c["val"]), c["key"][:-1])[np.repeat(np.arange(len(c["key"]) - 1),
                                                                         np.diff(c["key"]))]
    assert (np.abs(g["val"] - c["val"]) <= 128 * 2.0**-24 / np.sin(angle) * scale).all()


# the midpoints' Stokes noise on the vertices, four linearise events in flight: vertices with one event to 24 and (the
# fan's axis) 69, so every remainder of four; the right-hand side bit for bit
@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [lambda: kuhn_box(1, 1, 1, 5.0, seed=4), lambda: kuhn_box(3, 2, 4, 5.0, seed=4),
                                  lambda: fan(69)])
def test_midpoint_noise_forms(mesh):
    m = mesh()
    kw = dict(solver="CG", dt=1e-16, kT=4.11e-21, calc_noise=1, calc_stokes=1)
    b, o = lib.Blob(m, **kw), pyoracle.OracleBlob(m, threads=1, **kw)
    b.update(1)
    assert o.step(1) == 0
    assert np.array_equal(b.rhs()[:m.n_linear], o.rhs()[:m.n_linear])
