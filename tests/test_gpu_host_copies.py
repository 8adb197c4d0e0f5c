"""Copies of large pageable arrays through pinned slots: an OC update that cannot move (move 0) returns its densities
bit for bit, whatever the array's length against the staging line, the chunks and the slots, and its alignment; several
contexts at once; a context that goes and one that comes after it."""
import threading

import numpy as np
import pytest

from mycel_b200 import api

pytestmark = pytest.mark.gpu


def _through(ctx, n, offset=0, seed=0):
    rng = np.random.default_rng(n + seed)
    raw = rng.uniform(0.01, 1.0, n + offset)
    rho = raw[offset:]
    out, _ = api.oc_update(rho, -np.ones(n), np.ones(n), None, 0.5, 0.0, 1e-3, 1.0, 5, 1e-3, ctx=ctx)
    return np.array_equal(out, rho)


@pytest.mark.parametrize("n", [1, 131_071, 131_072, 131_073, 12 * 131_072 - 1, 12 * 131_072 + 1, 3_000_001])
def test_lengths(ctx, n):
    assert _through(ctx, n) and _through(ctx, n, offset=3)


def test_contexts_at_once_and_after_each_other():
    bad = []

    def work(k):
        for j in range(2):
            c = api.Context()
            for i in range(3):
                if not _through(c, 400_000 + 70_001 * k + i, seed=j):
                    bad.append((k, j, i))
            c.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
