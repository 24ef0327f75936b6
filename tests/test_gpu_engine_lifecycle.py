"""Engines made and closed in turn: each works, and what one held is free
again (whatever order its blocks are freed in)."""
import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import Engine, device_memory

pytestmark = pytest.mark.gpu


def test_what_an_engine_held_is_free_again():
    task = taskgen.negate_task(1)
    free, answers = [], []
    for _ in range(6):
        e = Engine(0, 2 << 30)
        s = e.solve(task, max_depth=4, sol_cap=64)
        answers.append((s.optimal_depth, s.programs))
        e.close()
        free.append(device_memory(0)[0])
    assert len(set(map(str, answers))) == 1
    assert min(free[1:]) >= free[0]


def test_engines_held_together_and_closed_in_another_order():
    task = taskgen.negate_task(1)
    before = None
    for _ in range(2):
        es = [Engine(0, 1 << 30) for _ in range(5)]
        got = [e.solve(task, max_depth=4, sol_cap=64).programs for e in es]
        for i in (3, 0, 4, 1, 2):
            es[i].close()
        assert all(g == got[0] for g in got)
        if before is not None:
            assert device_memory(0)[0] >= before
        before = device_memory(0)[0]
