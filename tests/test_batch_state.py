"""What a batch keeps between calls."""
import numpy as np
import pytest

from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import apply_shear, kuhn_box

pytestmark = pytest.mark.gpu

KW = dict(dt=1e-13, kT=4.11e-21, calc_noise=1)


def batch(cells=((12, 12, 12), (11, 12, 13), (3, 3, 3))):
    meshes = [kuhn_box(*c, 5.0, seed=4) for c in cells]
    return meshes, [apply_shear(m, 0.001) * (m.scale / 1.7e-10) for m in meshes]


def test_tuning_leaves_the_estimates(gpu):
    """A blob's first solve is the estimating one (Jacobi, several times the polynomial's iterations), and still is after
    tuning: what the tuner's solves have learnt is not kept."""
    meshes, x0 = batch()
    ref, bt = lib.Batch(meshes, **KW), lib.Batch(meshes, **KW)
    for b in (ref, bt):
        b.set_positions(np.concatenate(x0))
    bt.tune(solves=1)
    ref.update(1)
    bt.update(1)
    assert np.abs(ref.cg_iterations()[0] - bt.cg_iterations()[0]).max() <= 2


def test_what_config_reports_can_be_set(gpu):
    """config() and set_config() round-trip on chip and off it; both kernels, the streaming one with groups of several
    CTAs to a blob, take the blobs along the same trajectory (the mixed path's bound)."""
    meshes, x0 = batch(((12, 12, 12), (16, 15, 14), (9, 9, 9), (1, 1, 1)))
    bt = lib.Batch(meshes, **KW)
    assert bt.cg_kernel() == "sr_batch_kernel"
    chip = bt.config()
    bt.set_config(chip["cg_threads"], chip["threads_per_row"])
    assert bt.cg_kernel() == "sr_batch_kernel" and bt.config() == chip
    streams = [bt.rng_state(b) for b in range(len(meshes))]
    ends = []
    for shape in (None, (256, 4), (128, 1), (1024, 8)):
        if shape:
            bt.set_config(*shape)
            cfg = bt.config()
            assert bt.cg_kernel() == "cg_batch_kernel" and (cfg["cg_threads"], cfg["threads_per_row"]) == shape
            assert cfg["ctas"] >= 2 * len(meshes)
        bt.set_positions(np.concatenate(x0))
        for b, s in enumerate(streams):
            bt.set_rng_state(b, s)
        bt.update(3)
        ends.append([bt.pos(b) for b in range(len(meshes))])
    for b, p0 in enumerate(x0):
        move = np.abs(ends[0][b] - p0).max()
        for e in ends[1:]:
            assert np.abs(e[b] - ends[0][b]).max() < 1e-5 * move, b
    bt.set_config(chip["cg_threads"], chip["threads_per_row"])
    assert bt.cg_kernel() == "sr_batch_kernel" and bt.config() == chip
    bt.update(1)


# both sides of the plan's lines: four blobs to a block and five, and a blob of more rows than the chip holds
@pytest.mark.parametrize("cells,kernel", [([(2, 2, 2)] * 608, "sr_batch_kernel"), ([(2, 2, 2)] * 609, "cg_batch_kernel"),
                                          ([(1, 1, 1), (41, 42, 42)], "sr_batch_kernel"),
                                          ([(1, 1, 1), (43, 42, 41)], "cg_batch_kernel")])
def test_plan_of_the_solve(gpu, cells, kernel):
    box = {c: kuhn_box(*c, 5.0, seed=4) for c in set(cells)}
    bt = lib.Batch([box[c] for c in cells], **KW)
    assert bt.cg_kernel() == kernel
    bt.update(2)


def test_accuracy_of_the_solve_on_chip(gpu):
    """The batch's solutions are as near to FP64 as the streaming kernel's, whose q = V p is formed every iteration: the
    rms error of the moves over blobs of one block and of several, to a fifth (the spread over such sets)."""
    cells = [(4, 4, 4), (6, 6, 6), (7, 6, 7), (10, 10, 10), (14, 13, 14), (18, 18, 18)]
    meshes, x0 = batch(cells)
    bt = lib.Batch(meshes, **KW)
    streams = [bt.rng_state(b) for b in range(len(meshes))]
    exact = []
    for m, p, s in zip(meshes, x0, streams):
        f = lib.Blob(m, epsilon=1e-13, rng_state=s, **KW)
        f.set_state(pos=p)
        f.update(4)
        exact.append(f.pos())
    err = {}
    for kernel in ("sr_batch_kernel", "cg_batch_kernel"):
        if kernel == "cg_batch_kernel":
            bt.set_config(256, 4)
        assert bt.cg_kernel() == kernel
        bt.set_positions(np.concatenate(x0))
        for b, s in enumerate(streams):
            bt.set_rng_state(b, s)
        bt.update(4)
        err[kernel] = np.sqrt(np.mean([((bt.pos(b) - e) ** 2).sum() / ((e - x0[b]) ** 2).sum()
                                       for b, e in enumerate(exact)]))
    print(err)
    assert err["sr_batch_kernel"] <= 1.2 * err["cg_batch_kernel"]
