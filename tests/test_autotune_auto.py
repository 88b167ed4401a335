"""The autotuner does not pin a kernel that only the tuned batch wants: the
library's choice by the number of cells is a candidate, preferred unless a
named kernel is faster by more than timings scatter."""
import importlib

import pytest


class _FakeSolver:
    mech, variant = "fullchem", "fma"

    def set_launch(self, mode, threads, blocks_per_sm):
        self.launch = (mode, threads, blocks_per_sm)

    def set_chunk(self, cells):
        self.chunk = cells

    def set_row_scratch(self, shared):
        self.shared = shared


@pytest.fixture
def at():
    return importlib.import_module("geos-chem-gpu-hybrid_b200.autotune")


def test_automatic_entry_is_applied(at, pkg):
    s = _FakeSolver()
    at.apply(s, {"mode": "auto", "threads": 256, "blocks_per_sm": 0})
    assert s.launch == (pkg.AUTO, 256, 0) and s.chunk == 0


def test_automatic_choice_preferred_at_near_equal_speed(at):
    auto = at._score({"mode": "auto", "cells_per_s": 100.0})
    for mode in ("coop", "persistent", "plain"):
        assert at._score({"mode": mode, "cells_per_s": 102.0}) < auto
        assert at._score({"mode": mode, "cells_per_s": 110.0}) > auto
    for cands in (at.CANDIDATES, at.CHUNKED):
        settings = {c[1:] for c in cands if c[0] == "persistent" and c[4] == "global"}
        assert settings == {c[1:] for c in cands if c[0] == "auto"}


@pytest.mark.gpu
@pytest.mark.timeout(600)
def test_tuned_process_keeps_small_calls_fast(at, pkg):
    s = pkg.solver("fullchem", "fma")
    got = at.tune(s, pkg.workloads.plain_small(37888, seed=3), use_cache=False)
    best = {m: max(e["cells_per_s"] for e in got["table"] if (e["mode"] == "auto") == m) for m in (True, False)}
    named = got["mode"] != "auto"
    assert named == (max(at._score(e) for e in got["table"] if e["mode"] != "auto") >
                     max(at._score(e) for e in got["table"] if e["mode"] == "auto")), best
    if not named:
        assert s.workspace_slots(72) == 0 and s.workspace_slots(37888) > 0
    s.set_row_scratch(False)
    s.set_chunk(0)
    s.set_launch(pkg.PERSISTENT)
