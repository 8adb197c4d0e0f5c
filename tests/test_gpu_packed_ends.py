"""Packs in which some problems have ended, or wait for their next solve, while others still run, on both sides of the
lines that a pack's size is held against: its vector steps' CTAs an SM up to which kernels are launched as early
dependents (1), and the items an SM up to which a launch's steps and coarse products take more at once (3). Each problem
must come out with the bits of its run alone (tolerance 0)."""
import numpy as np
import pytest
import torch

from mycel_b200 import api
from mycel_b200 import workloads as W
from mycel_b200.model import OptimizerOptions
from test_gpu_packed import _alone, _same, _session

pytestmark = pytest.mark.gpu

BASE = OptimizerOptions(volume_fraction=0.3, filter_radius_mm=1.5, precision="mixed-mg", solver_tolerance_initial=1e-6,
                        solver_tolerance_final=1e-6, solver_max_iterations=20000)


GRIDS = {"early": ([(20, 10, 8), (26, 13, 9), (33, 17, 11)], 0.25),
         "few items": ([(64, 32, 20), (44, 22, 25), (50, 25, 33)], 0.4),
         "many items": ([(84, 42, 34), (64, 32, 40), (71, 35, 33)], 0.7)}


def _jobs(size):
    """(model, options): one iteration, five and three; a looser tolerance ends solves early as well."""
    grids, scale = GRIDS[size]
    jobs = []
    for (nx, ny, nz), iters, tol in zip(grids, (1, 5, 3), (1e-3, 1e-7, 1e-5)):
        jobs.append((W.cantilever(nx, ny, nz, e0=1.0, emin_ratio=1e-9, force=-1.0),
                     BASE.replace(max_iterations=iters, solver_tolerance_initial=tol, solver_tolerance_final=tol)))
    bp = next(b for b in W.batched_instances(count=16, seed=7, scale=scale) if len(b.load_cases) >= 3)
    jobs.append((bp.model, bp.options.replace(max_iterations=2, precision="mixed-mg", separate_load_cases=True)))
    return jobs


@pytest.mark.parametrize("size", list(GRIDS))
def test_problems_that_end_at_different_times(ctx, size):
    jobs = _jobs(size)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ctas = sum(-(-(m.total_dofs // 4) // 1024) * (len(m.loads) if o.separate_load_cases else 1) for m, o in jobs)
    rows = sum(-(-np.prod([(n + 1) // 2 + 1 for n in (m.grid.nx, m.grid.ny, m.grid.nz)]) // 64) for m, _ in jobs[:3])
    assert (ctas <= sms) == (size == "early")
    assert (ctas > 3 * sms) == (rows > 3 * sms) == (size == "many items")
    alone = [_alone(ctx, m, o, o.max_iterations) for m, o in jobs]
    made = [_session(ctx, m, o) for m, o in jobs]
    try:
        before = ctx.packed_count
        out = api.SimpSession.run_many([s for _, s in made])
        reads = [s.read() for _, s in made]
        assert ctx.packed_count > before
    finally:
        for p, s in made:
            s.close()
            p.close()
    for k, (ra, da) in enumerate(alone):
        _same(ra, da, out[k], reads[k])
