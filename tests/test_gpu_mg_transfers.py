"""The multigrid transfers on both sides of the line between a thread per component and a thread per pair of nodes
(262,144 pairs): a level below it for one case and above it for two. Two cases together must give the bits of each
alone."""
import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200.model import FeModel, StaticAnalysisOptions
from test_gpu_mg_small_levels import _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(96, 64, 64), (97, 63, 62)])
def test_two_cases_equal_each_alone(ctx, shape):
    m = _model(*shape, 2)
    o = StaticAnalysisOptions(tolerance=1e-8, max_iterations=5000, precision="mixed-mg")
    for k, r in enumerate(api.StaticAnalysis.run_cases(m, o, ctx)):
        one = FeModel(m.grid, m.domain, m.material, m.fixed_dofs, [m.loads[k]], element_density=m.element_density)
        alone = api.StaticAnalysis.run(one, o, ctx, reactions=False, von_mises=False)
        assert r.solver_info.final_residual <= 1e-8
        assert np.array_equal(r.u, alone.u)
