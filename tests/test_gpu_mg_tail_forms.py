"""The two forms of the cluster kernel of the small multigrid levels against each other: sixteen CTAs with the levels in
their shared memory, and eight with the vectors in global memory (what a device takes that cannot hold the first;
MYCEL_MG_TAIL=global). Every sum is formed in the same order, so the solves must have the same bits, alone, with load
cases together and packed; the first form also when it is run again and again (its CTAs write into one another's
memory)."""
import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200 import workloads as W
from mycel_b200.model import OptimizerOptions, StaticAnalysisOptions
from test_gpu_mg_small_levels import _model
from test_gpu_packed import _same, _session

pytestmark = pytest.mark.gpu
O = StaticAnalysisOptions(tolerance=1e-8, max_iterations=5000, precision="mixed-mg")


def _solve(ctx, m, cases):
    before = ctx.launch_count
    r = api.StaticAnalysis.run_cases(m, O, ctx) if cases > 1 else [api.StaticAnalysis.run(m, O, ctx, reactions=False,
                                                                                       von_mises=False)]
    assert all(x.solver_info.final_residual <= 1e-8 for x in r)
    return np.stack([x.u for x in r]), [x.solver_info.iterations for x in r], ctx.launch_count - before


@pytest.mark.parametrize("shape,cases", [((64, 32, 40), 1), ((64, 32, 40), 4), ((5, 4, 3), 2), ((37, 23, 11), 8),
                                         ((131, 9, 7), 1)])
def test_shared_memory_form_equals_global_memory_form(ctx, monkeypatch, shape, cases):
    m = _model(*shape, cases)
    _solve(ctx, m, cases)  # the product is tuned on a grid's first solve
    u, its, launches = _solve(ctx, m, cases)
    monkeypatch.setenv("MYCEL_MG_TAIL", "global")
    ug, itsg, launches_g = _solve(ctx, m, cases)
    assert its == itsg and np.array_equal(u, ug)
    if shape == (64, 32, 40):  # 17x9x11 nodes go to the cluster in global memory only: the forms did differ
        assert launches > launches_g


def test_shared_memory_form_again_and_again(ctx):
    m = _model(40, 30, 20, 1)
    u = _solve(ctx, m, 1)[0]
    for _ in range(20):
        assert np.array_equal(_solve(ctx, m, 1)[0], u)


def test_packed_problems_of_both_forms(ctx, monkeypatch):
    o = OptimizerOptions(volume_fraction=0.3, filter_radius_mm=1.5, max_iterations=2, precision="mixed-mg",
                         solver_tolerance_initial=1e-6, solver_tolerance_final=1e-6, solver_max_iterations=20000)
    models = [W.cantilever(n, 12, 8, e0=1.0, emin_ratio=1e-9, force=-1.0) for n in (24, 33, 20)]

    def run(forms):
        made = []
        try:
            for m, form in zip(models, forms):
                monkeypatch.setenv("MYCEL_MG_TAIL", form)
                made.append(_session(ctx, m, o))
                made[-1][1].step()  # builds the hierarchy
            return api.SimpSession.run_many([s for _, s in made]), [s.read() for _, s in made]
        finally:
            for p, s in made:
                s.close()
                p.close()

    ra, da = run(["", "", ""])
    rb, db = run(["", "global", "global"])
    for k in range(3):
        _same(ra[k], da[k], rb[k], db[k])
