"""The long stages of solves that share the GPU (a server's): launched in
ranges, with the answers of the same solve alone, at most a bounded time later,
and a batch's stages not later at all."""
import random

import pytest

from pca_gb300.pcalib import make_task

pytestmark = pytest.mark.gpu
M = 0xFFFF


def two_inputs(f, seed, tests=27):
    rng = random.Random(seed)
    rows = [[rng.randrange(1 << 16) for _ in range(2)] for _ in range(tests)]
    return make_task("two", rows, [f(*r) & M for r in rows])


def both(engine, tasks, **kw):
    """The batch alone (twice: the first settles the engine's costs) and shared."""
    for _ in range(2):
        alone = engine.solve_batch(tasks, **kw)
    shared = engine.solve_batch(tasks, shared_gpu=True, **kw)
    for a, s in zip(alone, shared):
        assert (s.optimal_depth, s.total_solutions, s.programs, s.candidates, s.evaluations) == \
               (a.optimal_depth, a.total_solutions, a.programs, a.candidates, a.evaluations)
    return alone, shared


def test_a_batch_of_open_tasks_is_not_slowed(engine):
    """Each task's stage is short; their sum is not."""
    tasks = [two_inputs(max, s) for s in range(40)]
    alone, shared = both(engine, tasks, max_depth=4, first_only=True, sol_cap=1)
    assert all(s.optimal_depth == -1 for s in shared)
    assert shared[0].gpu_ms_suffix < 4 * alone[0].gpu_ms_suffix + 10


@pytest.mark.parametrize("first_only", [True, False])
def test_one_long_stage_steps_back_for_a_bounded_time(engine, first_only):
    tasks = [two_inputs(max, 0)]
    alone, shared = both(engine, tasks, max_depth=5, first_only=first_only, split_depth=2,
                         sol_cap=64)
    assert shared[0].optimal_depth == -1
    assert shared[0].gpu_ms_suffix < 2 * alone[0].gpu_ms_suffix + 900


# optimal at depth 5, from a level whose stage takes longer than one range
LONG = [lambda x, y: ((x * y) ^ (x + y)) - (x & y), lambda x, y: ((x + y) * y ^ x) - (x & y)]


@pytest.mark.parametrize("first_only", [True, False])
@pytest.mark.parametrize("k", range(len(LONG)))
@pytest.mark.parametrize("split", [2, 3])
def test_solutions_of_ranges_are_the_stage_s(engine, k, split, first_only):
    tasks = [two_inputs(LONG[k], 5, 20)]
    alone, shared = both(engine, tasks, max_depth=5, first_only=first_only, split_depth=split,
                         sol_cap=256)
    assert shared[0].optimal_depth == 5 and shared[0].programs


def test_a_batch_of_long_stages(engine):
    """Groups of one task and of several, longer than a range."""
    tasks = [two_inputs(max, 3), two_inputs(LONG[0], 5, 20), two_inputs(lambda x, y: x + y, 1),
             two_inputs(min, 4)]
    alone, shared = both(engine, tasks, max_depth=5, first_only=True, split_depth=2, sol_cap=4)
    assert [s.optimal_depth for s in shared] == [-1, 5, 1, -1]
    assert shared[0].gpu_ms_suffix < 2 * alone[0].gpu_ms_suffix + 900
