"""Contexts, problems, filters and sessions given back in any order (a garbage collector finalises the members of a
cycle in no particular one, so does the end of a program): the library must be asked to free each once, and nothing
after what it belongs to. The library is a stand-in that records the calls."""
import gc
import itertools

import numpy as np
import pytest

from mycel_b200 import api
from mycel_b200 import workloads as W
from mycel_b200.model import OptimizerOptions


class _Lib:
    """Hands out numbers as handles and checks every handle that it is given back."""

    def __init__(self):
        self.next = itertools.count(100)
        self.live = {}  # handle -> its parent
        self.log = []

    def _make(self, parent, out):
        h = next(self.next)
        assert parent is None or parent in self.live, "made on a freed parent"
        self.live[h] = parent
        out._obj.value = h
        return 0

    def _free(self, kind, h):
        assert h in self.live, f"{kind} freed twice, or after what it belongs to"
        for c in [c for c, p in self.live.items() if p == h]:
            assert kind == "problem" and self.kinds[c] == "session", f"{kind} freed before what belongs to it"
            del self.live[c]  # a problem ends its sessions
        del self.live[h]
        self.log.append(kind)
        return 0

    def load(self):
        return self

    kinds = {}

    def mycel_ctx_create(self, device, out):
        return self._make(None, out)

    def mycel_problem_create(self, ctx, *rest):
        return self._make(ctx, rest[-1])

    def mycel_filter_create(self, p, rmin, out):
        return self._make(p, out)

    def mycel_simp_begin(self, p, so, out):
        r = self._make(p, out)
        self.kinds[out._obj.value] = "session"
        return r

    def mycel_ctx_destroy(self, h):
        return self._free("context", h)

    def mycel_problem_destroy(self, h):
        return self._free("problem", h)

    def mycel_filter_destroy(self, h):
        return self._free("filter", h)

    def mycel_simp_end(self, h):
        return self._free("session", h)


@pytest.fixture
def lib(monkeypatch):
    lib = _Lib()
    errors = []
    monkeypatch.setattr(api.L, "load", lambda: lib)
    free = lib._free

    def checked(kind, h):  # __del__ swallows exceptions
        try:
            return free(kind, h)
        except AssertionError as e:
            errors.append(str(e))
            return 0

    lib._free = checked
    lib.errors = errors
    return lib


def _make():
    ctx = api.Context(0)
    prob = api.Problem(W.cantilever(3, 2, 2), ctx)
    flt = api.DensityFilter(prob, 1.5)
    sess = api.SimpSession(prob, OptimizerOptions())
    return dict(context=ctx, problem=prob, filter=flt, session=sess)


@pytest.mark.parametrize("order", list(itertools.permutations(["context", "problem", "filter", "session"])))
def test_closed_in_any_order(lib, order):
    made = _make()
    for k in order:
        made[k].close()
    made.clear()
    gc.collect()
    assert not lib.errors and not lib.live, (lib.errors, lib.log)


@pytest.mark.parametrize("order", list(itertools.permutations(["context", "problem", "filter", "session"])))
def test_collected_in_any_order(lib, order):
    """Finalisers of a cycle's members run in the collector's order: here one after the other, as given."""
    made = _make()
    for k in order:
        made[k].__del__()
    made.clear()
    gc.collect()
    assert not lib.errors and not lib.live, (lib.errors, lib.log)


def test_collected_as_a_cycle(lib):
    for n in range(6):
        made = list(_make().values())
        made = made[n % 4:] + made[:n % 4]
        made.append(made)
        del made
        gc.collect()
    assert not lib.errors and not lib.live, (lib.errors, lib.log)
