"""The plain PCG's kernels at the edges of their tiles, bit for bit against the oracle: K x for node rows around the
staged span (one range of rows up to 130 nodes, three beyond), one to several chunks a plane, and whole iterations
(direction formed in the product, lane chains, block sums) for DOF counts of every remainder mod 4, one block,
blocks that end on a boundary, and several."""
import numpy as np
import pytest

from mycel_b200 import api
from models import carved_model, tiny_test_model

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (2, 1, 3), (30, 10, 4), (63, 3, 2), (127, 2, 1), (128, 1, 2), (129, 2, 2), (130, 3, 1), (131, 1, 1),
         (260, 4, 2), (15, 15, 31), (40, 20, 10), (34, 22, 11)]


@pytest.mark.parametrize("shape", GRIDS)
def test_product_and_iterations(oracle, ctx, shape):
    nx, ny, nz = shape
    m = carved_model(nx, ny, nz, seed=nx + ny, frac=0.1) if nx > 2 else tiny_test_model(nx, ny, nz)
    oracle.set_modes(lane_mode=0, threads=8)
    om, pr = oracle.Model(m), api.Problem(m, ctx)
    x = np.random.default_rng(nx).normal(size=m.total_dofs)
    assert np.array_equal(pr.apply_k(x), om.apply_k(x))
    b = om.forces() * (om.constrained() == 0)
    for x0 in (None, 1e-3 * x * (om.constrained() == 0)):
        for its in (1, 2, 37):  # odd and even ends of the alternating direction buffers, over a chunk's end
            ug, rg = pr.pcg_solve(b, x0=x0, tol=1e-14, max_iterations=its)
            uo, ro = om.pcg_solve(b, x0=x0, tol=1e-14, max_iter=its)
            assert rg.iterations == ro.iterations and rg.final_residual == ro.final_residual
            assert np.array_equal(ug, uo)
