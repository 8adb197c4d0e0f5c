"""Solves on a GPU whose memory another allocator holds: a solve that runs out part-way through a workspace raises, and
the same problem solves once there is room again, with the bits of a problem that never ran out. The memory is handed
back in steps smaller than a vector, so the workspaces are left unfinished in several places."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
import numpy as np, torch
from mycel_b200 import api, workloads as W
from mycel_b200.model import OutOfMemoryError
form, MB = sys.argv[1], 1 << 20
model = lambda *n: W.cantilever(*n, e0=1.0, emin_ratio=1e-9, force=-1.0)
ctx = api.Context(0)
def solve(prob):
    return prob.pcg_solve(prob.forces(), tol=1e-6, max_iterations=40, precision=form)
small = api.Problem(model(40, 20, 16), ctx)  # the kernels are loaded while there is room
solve(small)
prob = api.Problem(model(144, 72, 60), ctx)  # 1.9 million DOFs: 15.5 MB a vector
torch.cuda.synchronize()
held = []
while len(held) < 100000:  # all that is free: most of it at once, then pieces that are handed back one by one
    free = torch.cuda.mem_get_info()[0]
    try:
        held.append(torch.cuda.caching_allocator_alloc(free - 800 * MB if free > 1000 * MB else 12 * MB))
    except torch.OutOfMemoryError:
        break
failed = 0
while True:
    try:
        x, r = solve(prob)
        break
    except OutOfMemoryError:
        failed += 1
        torch.cuda.caching_allocator_delete(held.pop())
        torch.cuda.empty_cache()
while held:
    torch.cuda.caching_allocator_delete(held.pop())
torch.cuda.empty_cache()
y, s = solve(api.Problem(model(144, 72, 60), api.Context(0)))
assert np.array_equal(x, y) and r.iterations == s.iterations
print("failed", failed)
"""


@pytest.mark.parametrize("form", ["fp64", "mixed", "fp64f", "mixed-mg"])
def test_a_solve_that_ran_out_can_be_repeated(form):
    r = subprocess.run([sys.executable, "-c", CODE, form], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) >= 2, "too little was held back for the solve to run out part-way"
