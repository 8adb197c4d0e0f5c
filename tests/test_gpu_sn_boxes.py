"""MakeWellComposed (SurfaceNetsExtractor.cs:352-435) in waves of skewed boxes: the sequential sweep's mask, density,
passes and resolutions at the edges of boxes (32 x 16 x 16 in x + y + 2z, y + z, z) and of mask words, for fields with
something to resolve nearly everywhere, in few boxes, and in one place."""
import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200.model import GridSpec
from meshtools import saddle_field

pytestmark = pytest.mark.gpu


def _field(kind, nx, ny, nz):
    if kind == "dense":
        return saddle_field(nx, ny, nz, seed=nx + ny)
    if kind == "sparse":
        return saddle_field(nx, ny, nz, seed=nz, p=0.04)
    # a diagonal chain of voxels through the whole grid: each resolution makes the next ones
    d = np.full((nz, ny, nx), 0.1, np.float32)
    m = max(nx, ny, nz)
    for k in range(m):
        d[k * nz // m, k * ny // m, k * nx // m] = 0.6 + 0.3 * (k % 7) / 7
    return d.ravel()


@pytest.mark.parametrize("kind", ["dense", "sparse", "chain"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (29, 13, 14), (30, 15, 16), (32, 16, 15), (33, 17, 17), (64, 33, 31),
                                   (7, 90, 40), (130, 5, 70)])
def test_boxes_match_the_sequential_sweep(oracle, ctx, kind, shape):
    nx, ny, nz = shape
    d = _field(kind, nx, ny, nz)
    pos, idx, info = oracle.surface_nets(nx, ny, nz, d, threshold=0.5)
    m = api.SurfaceNetsExtractor.extract(GridSpec(nx, ny, nz, 1.0, (0.0, 0.0, 0.0)), d, 0.5, ctx=ctx)
    assert (m.passes, m.changes) == (info["passes"], info["changes"])
    assert m.positions.shape == pos.shape and np.array_equal(m.positions.view(np.uint32), pos.view(np.uint32))
    assert np.array_equal(m.indices, idx)
