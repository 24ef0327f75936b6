"""A level whose distinct columns outnumber the ids is built once more
without them, from either of the places that read the build's status (one
round trip for a level that fits an eighth of the arena, two for a larger
one): its levels, counters and programs are those of the ids."""
import ctypes
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import OEP_EXACT, OEP_EXACT_LIVE, Engine, make_task

pytestmark = pytest.mark.gpu


def limit(engine, most):
    fn = engine.lib.pcagb_internal_limit_ids
    fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_uint64], None
    fn(engine.h, most)


def answers(s):
    return (s.optimal_depth, s.total_solutions, s.programs, s.level_survivors, s.level_children,
            s.tried, s.pruned_cum, s.candidates, s.insert_launches, s.insert_children)


def task(inputs, tests, seed):
    rng = random.Random(seed)
    rows = [[rng.randrange(1 << 16) for _ in range(inputs)] for _ in range(tests)]
    return make_task("ids", rows, [rng.randrange(1 << 16) for _ in rows])


# two inputs: 202,365 children at level 2, which an eighth of 600 MB does not hold
@pytest.mark.parametrize("arena", [600 << 20, 4 << 30])
@pytest.mark.parametrize("mode", [OEP_EXACT, OEP_EXACT_LIVE])
@pytest.mark.parametrize("tests", [3, 16, 32])
def test_levels_of_a_rebuild(arena, mode, tests):
    eng = Engine(0, arena)
    try:
        t = task(2, tests, tests)
        want = eng.solve(t, max_depth=2, oep_mode=mode, count_levels=True)
        for most in (1, 64, 1000):
            limit(eng, most)
            got = eng.solve(t, max_depth=2, oep_mode=mode, count_levels=True)
            assert answers(got) == answers(want)
            # it is the rebuild that answered
            assert got.kernel_launches > want.kernel_launches
        limit(eng, (1 << 64) - 1)
        again = eng.solve(t, max_depth=2, oep_mode=mode, count_levels=True)
        assert answers(again) == answers(want) and again.kernel_launches == want.kernel_launches
    finally:
        eng.close()


def test_a_search_with_every_level_rebuilt():
    """Full and lean levels, and a batch."""
    eng = Engine(0, 16 << 30)
    try:
        power2 = taskgen.is_power2_task(1)
        mix = [t for _, t in taskgen.poisson_stream(12, rate=100.0, seed=21)]
        for f in (lambda: [eng.solve(power2, max_depth=4, split_depth=3)],
                  lambda: [eng.solve(power2, max_depth=3, count_levels=True)],
                  lambda: eng.solve_batch(mix, max_depth=4, split_depth=2, sol_cap=8)):
            limit(eng, (1 << 64) - 1)
            want = [answers(s) for s in f()]
            limit(eng, 2000)
            assert [answers(s) for s in f()] == want
    finally:
        eng.close()
