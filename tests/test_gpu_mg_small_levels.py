"""The multigrid levels that share one cluster launch with their data in shared memory, against the launches of a
kernel per phase: the same solve with load cases together (whose room decides from which level on the cluster kernel
runs, and how many cases it takes at once) and alone must give the same bits, and the residual must be met.

Grids: a finest small level that one case fits and several do not, one that does not fit with its stencil, only the
coarsest level, long thin levels, odd counts on every axis, and eight cases (the most solved together)."""
import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200.model import FeMaterial, FeModel, GridSpec, LoadCase, StaticAnalysisOptions, SurfacePatch

pytestmark = pytest.mark.gpu


def _model(nx, ny, nz, cases):
    rng = np.random.default_rng(nx + ny + nz)
    g = GridSpec(nx, ny, nz, 1.0)
    fixed = FeModel.fix_dofs([g.node_index(0, j, k) for k in range(nz + 1) for j in range(ny + 1)])
    loads = [LoadCase(SurfacePatch([g.node_index(nx, int(rng.integers(ny + 1)), int(rng.integers(nz + 1)))], [1.0]),
                      tuple(rng.normal(size=3))) for _ in range(cases)]
    return FeModel(g, np.ones(g.total_elements), FeMaterial(1.0, 0.3, 1e-6), fixed, loads,
                   element_density=rng.uniform(0.3, 1.0, g.total_elements))


@pytest.mark.parametrize("shape,cases", [((64, 32, 40), 4), ((50, 46, 44), 2), ((5, 4, 3), 3), ((300, 5, 4), 2),
                                         ((37, 23, 11), 8), ((27, 27, 27), 5)])
def test_together_equals_alone(ctx, shape, cases):
    m = _model(*shape, cases)
    o = StaticAnalysisOptions(tolerance=1e-8, max_iterations=5000, precision="mixed-mg")
    together = api.StaticAnalysis.run_cases(m, o, ctx)
    for k, r in enumerate(together):
        one = FeModel(m.grid, m.domain, m.material, m.fixed_dofs, [m.loads[k]], element_density=m.element_density)
        alone = api.StaticAnalysis.run(one, o, ctx, reactions=False, von_mises=False)
        assert r.solver_info.final_residual <= 1e-8 and r.solver_info.fallback_iterations == 0
        assert r.solver_info.iterations == alone.solver_info.iterations
        assert np.array_equal(r.u, alone.u)
