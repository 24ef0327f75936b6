"""The last positions over value forms (a lane per state) against the
warp-per-item kernels that evaluate every class: the same solving programs
in the same order, the same counters, from every split (suffix depths 1 to
3, the root included), at test counts around the four tests of a probe and
the 16- and 32-test widths, with no, one and two inputs, with and without
the pruner."""
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import OEP_EXACT_LIVE, OEP_NONE, make_task

pytestmark = pytest.mark.gpu


def task(inputs, tests, length, seed):
    rng = random.Random(seed)
    rows = [[rng.choice([0, 1, 0xFFFF, 0x8000, rng.randrange(16), rng.randrange(1 << 16)])
             for _ in range(inputs)] for _ in range(tests)]
    prog = taskgen.random_program(rng, length)
    return make_task("forms", rows, [taskgen.run_program(prog, r)[prog[-1][1]] for r in rows])


def same(a, b):
    assert a.optimal_depth == b.optimal_depth
    assert a.total_solutions == b.total_solutions
    assert a.programs == b.programs
    assert a.candidates == b.candidates and a.evaluations == b.evaluations
    assert a.evaluations_run == b.evaluations_run


@pytest.mark.parametrize("mode", [OEP_EXACT_LIVE, OEP_NONE])
@pytest.mark.parametrize("tests", [1, 2, 3, 4, 5, 16, 17, 32])
@pytest.mark.parametrize("inputs", [0, 1, 2])
def test_same_sets_as_the_warp_kernels(engine, inputs, tests, mode):
    for seed in range(6):
        t = task(inputs, tests, 3 + seed % 3, 1000 * inputs + 10 * tests + seed)
        for split in (0, 1, 2):
            want = engine.solve(t, max_depth=3 if split else 2, split_depth=split, oep_mode=mode,
                                sol_cap=1 << 14, suffix_chunk=16)
            got = engine.solve(t, max_depth=3 if split else 2, split_depth=split, oep_mode=mode,
                               sol_cap=1 << 14, suffix_chunk=1024)
            same(got, want)
            if split == 2:
                one = engine.solve(t, max_depth=3, split_depth=2, oep_mode=mode, sol_cap=1 << 14,
                                   suffix_chunk=1)
                same(got, one)


@pytest.mark.parametrize("split", [0, 1, 2])
def test_depth3_first_programs(engine, split):
    """Optimal depth 3 with two inputs: suffix depths 3, 2 and 1 over
    thousands of states."""
    found = 0
    for seed in range(400):
        t = task(2, 20, 4, 90000 + seed)
        auto = engine.solve(t, max_depth=3, first_only=True, sol_cap=1)
        if auto.optimal_depth != 3:
            continue
        found += 1
        got = engine.solve(t, max_depth=3, split_depth=split, sol_cap=1 << 14)
        want = engine.solve(t, max_depth=3, split_depth=split, sol_cap=1 << 14,
                            suffix_chunk=16 if split < 2 else 1)
        same(got, want)
        if found == 6:
            break
    assert found >= 3


@pytest.mark.parametrize("value", [0, 1, 6, 255, 256, 0xFFFF, 0xFFFE, 0xFFFD, 0xFFFC, 0x8000])
@pytest.mark.parametrize("inputs", [0, 1, 2])
def test_constant_targets(engine, inputs, value):
    """Constants: LDI, zero and an ADDI, longer ones; the copies and zeros
    that the forms leave out are on these programs' way."""
    rng = random.Random(value)
    rows = [[rng.randrange(1 << 16) for _ in range(inputs)] for _ in range(9)]
    t = make_task("constant", rows, [value] * 9)
    for mode in (OEP_EXACT_LIVE, OEP_NONE):
        for split in (0, 1, 2):
            depth = 3 if split else 2
            got = engine.solve(t, max_depth=depth, split_depth=split, oep_mode=mode, sol_cap=1 << 14)
            want = engine.solve(t, max_depth=depth, split_depth=split, oep_mode=mode,
                                sol_cap=1 << 14, suffix_chunk=16 if split < 2 else 1)
            same(got, want)
    first = engine.solve(t, max_depth=3, first_only=True, sol_cap=1)
    every = engine.solve(t, max_depth=3, split_depth=0, sol_cap=1 << 14, suffix_chunk=16)
    assert (first.optimal_depth, first.programs) == (every.optimal_depth, every.programs[:1])
