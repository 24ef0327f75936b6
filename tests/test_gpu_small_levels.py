"""Level builds whose bookkeeping runs in one block and one clearing launch
(up to 2^20 children, 16,384 parents) against larger ones, and where the arena
is too small to lay their scratch out side by side: the same levels, counters
and programs, or the same refusal."""
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import OEP_EXACT_LIVE, OEP_NONE, Engine, EngineError, make_task

pytestmark = pytest.mark.gpu


def task(inputs, tests, seed):
    rng = random.Random(seed)
    rows = [[rng.choice([0, 1, 0xFFFF, 0x8000, rng.randrange(16), rng.randrange(1 << 16)])
             for _ in range(inputs)] for _ in range(tests)]
    prog = taskgen.random_program(rng, 6)
    return make_task("levels", rows, [taskgen.run_program(prog, r)[prog[-1][1]] for r in rows])


def facts(s):
    return (s.optimal_depth, s.total_solutions, s.programs, s.candidates, s.evaluations,
            list(s.level_children), list(s.level_survivors), s.tried, s.pruned_cum)


@pytest.mark.parametrize("mode", [OEP_EXACT_LIVE, OEP_NONE])
@pytest.mark.parametrize("inputs,tests", [(0, 1), (1, 16), (1, 17), (2, 32)])
def test_levels_from_every_split(engine, inputs, tests, mode):
    """Counters and levels of a count-mode solve (every level built, one of
    them past the small sizes with two inputs) are those of the levels built
    from other splits, and of a second solve on the same engine."""
    for seed in range(4):
        t = task(inputs, tests, 100 * inputs + seed)
        depth = 2 if mode == OEP_NONE else 3
        want = engine.solve(t, max_depth=depth, count_levels=True, oep_mode=mode, sol_cap=64)
        again = engine.solve(t, max_depth=depth, count_levels=True, oep_mode=mode, sol_cap=64)
        assert facts(again) == facts(want)
        for split in range(depth):
            s = engine.solve(t, max_depth=depth, split_depth=split, oep_mode=mode, sol_cap=64)
            # (the counters' levels hold one program of each state)
            assert s.optimal_depth == want.optimal_depth
            assert s.programs[:1] == want.programs[:1]
            # a level is built only when its depth is reached (0: it was not)
            for got, whole in ((s.level_survivors, want.level_survivors),
                               (s.level_children, want.level_children)):
                assert all(g in (0, w) for g, w in zip(got, whole))


@pytest.mark.parametrize("inputs", [1, 2])
def test_small_arenas(engine, inputs):
    """From an arena in which nothing fits to one in which all does, a solve
    through level 2 is refused or gives the same answer, and what fits an
    arena fits a larger one."""
    t = task(inputs, 32, 7)
    want = facts(engine.solve(t, max_depth=3, split_depth=2, sol_cap=64))
    fitted = False
    for kb in (256, 512, 1024, 2048, 3072, 4096, 6144, 8192, 12288, 16384, 24576, 32768, 65536,
               131072):
        eng = Engine(0, kb << 10)
        try:
            got = facts(eng.solve(t, max_depth=3, split_depth=2, sol_cap=64))
        except EngineError:
            assert not fitted
            continue
        finally:
            eng.close()
        assert got == want
        fitted = True
    assert fitted
