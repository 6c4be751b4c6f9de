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
