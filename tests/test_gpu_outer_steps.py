"""The outer steps of the iterative forms and their sums over CTAs: one CTA, a few, and both sides of the line
(3 CTAs an SM) between several loads in flight and one. The FP64 factorised form against the plain one, the multigrid
forms against the FP64 factorised one, at the tolerances stated for solves to 1e-10: compliance to 1e-8, u to 1e-6."""
import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200.model import FeMaterial, FeModel, GridSpec, LoadCase, StaticAnalysisOptions, SurfacePatch

pytestmark = pytest.mark.gpu


def _model(nx, ny, nz):
    rng = np.random.default_rng(nx * ny + nz)
    g = GridSpec(nx, ny, nz, 1.0)
    fixed = FeModel.fix_dofs([g.node_index(0, j, k) for k in range(nz + 1) for j in range(ny + 1)])
    tip = [g.node_index(nx, j, 0) for j in range(ny + 1)]
    load = LoadCase(SurfacePatch(tip, [1.0 / len(tip)] * len(tip)), (0.1, 0.2, -1.0))
    return FeModel(g, np.ones(g.total_elements), FeMaterial(1.0, 0.3, 1e-6), fixed, [load],
                   element_density=rng.uniform(0.5, 1.0, g.total_elements))


@pytest.mark.parametrize("shape,forms", [((2, 1, 1), ("fp64", "fp64f", "mg", "mixed-mg")),
                                         ((33, 18, 11), ("fp64", "fp64f", "mg", "mixed-mg")),
                                         ((100, 77, 75), ("fp64f", "mg", "mixed-mg")),
                                         ((100, 77, 76), ("fp64f", "mg", "mixed-mg"))])
def test_forms_agree(ctx, shape, forms):
    m = _model(*shape)
    ref = None
    for f in forms:
        o = StaticAnalysisOptions(tolerance=1e-10, max_iterations=20000, precision=f)
        r = api.StaticAnalysis.run(m, o, ctx, reactions=False, von_mises=False)
        assert r.solver_info.final_residual <= 1e-10
        if ref is None:
            ref = r
        assert abs(r.compliance - ref.compliance) <= 1e-8 * ref.compliance
        assert np.max(np.abs(r.u - ref.u)) <= 1e-6 * np.max(np.abs(ref.u))
