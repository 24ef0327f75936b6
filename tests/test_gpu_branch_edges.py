"""Branch mode at the edges of its test widths, against the CPU restatement of
the walk with the exact pruner (oracle.enumerate_branch): counters, programs
and their order, on tasks with many solutions (the walk stops at the 100th,
inside a level) and with few, with divisions that fault; and the last position
without its level finds the same programs."""
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import make_task

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tests", [1, 2, 3, 4, 8, 15, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("inputs", [1, 2])
def test_walk_and_programs(engine, inputs, tests):
    from oracle import oracle as O
    for seed in range(4):
        rng = random.Random(1000 * inputs + 10 * tests + seed)
        rows = [[rng.choice([0, 1, 3, 0xFFFF, 0x8000, rng.randrange(1 << 16)])
                 for _ in range(inputs)] for _ in range(tests)]
        if seed == 0:      # signed division by the first input, 0 where it faults
            signed = lambda v: v - 0x10000 if v & 0x8000 else v  # noqa: E731
            out = [int(5 / signed(r[0])) & 0xFFFF if r[0] else 5 for r in rows]
        else:
            prog = taskgen.random_program(rng, seed + 1)
            out = [taskgen.run_program(prog, r)[prog[-1][1]] for r in rows]
        task = make_task("edges", rows, out)
        r, progs = O.enumerate_branch(task, 2, O.EXACT)
        sol = engine.solve_branch(task, max_depth=2, sol_cap=100)
        assert sol.optimal_depth == r.optimal_depth
        last = r.optimal_depth if r.optimal_depth >= 0 else 2
        assert sol.tried == [r.tried[k] for k in range(last + 1)]
        assert sol.pruned_cum == [r.pruned_cum[k] for k in range(last + 1)]
        assert sol.programs == progs
        if r.optimal_depth >= 1:
            direct = engine.solve_branch(task, max_depth=2, last_level_max_children=0)
            assert (direct.optimal_depth, direct.programs) == (r.optimal_depth, progs)
            first = engine.solve_branch(task, max_depth=2, first_only=True, sol_cap=1)
            assert (first.optimal_depth, first.programs) == (r.optimal_depth, progs[:1])
