"""The solutions a caller takes: a list of at most sol_cap programs is the
beginning of the whole list, whatever the cap cuts (a prefix's last
positions share one read result), and the score of a program does not depend
on what ran before it in the same machine."""
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import OEP_EXACT, OEP_EXACT_LIVE, OEP_NONE, PCALib, make_task


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [OEP_EXACT_LIVE, OEP_NONE, OEP_EXACT])
@pytest.mark.parametrize("split", [0, 1, 2])
def test_a_capped_list_is_the_beginning_of_the_whole(engine, split, mode):
    # solved at depths 1, 2 and 3 by a handful to thousands of programs
    for task in (make_task("double", [[1], [2]], [2, 4]),
                 make_task("two", [[3, 5], [3, 9], [4, 1]], [8, 12, 5]),
                 make_task("mix", [[1], [2], [7]], [14, 28, 98])):
        whole = engine.solve(task, max_depth=3, split_depth=split, oep_mode=mode, sol_cap=1 << 17)
        assert len(whole.programs) == whole.total_solutions or mode == OEP_EXACT
        assert len(set(map(tuple, whole.programs))) == len(whole.programs)
        n = len(whole.programs)
        for cap in {0, 1, 2, 3, n // 3, n - 1, n, n + 1}:
            part = engine.solve(task, max_depth=3, split_depth=split, oep_mode=mode,
                                sol_cap=max(cap, 0))
            assert part.programs == whole.programs[:max(cap, 0)]
            assert part.total_solutions == whole.total_solutions
            assert part.optimal_depth == whole.optimal_depth


def test_scores_do_not_depend_on_the_tests_before():
    """Programs with loads, stores, calls and jumps: passing tests counted
    together are those counted one test at a time."""
    lib = PCALib()
    rng = random.Random(5)
    checked = 0
    for _ in range(3000):
        prog = [rng.randrange(0x19) << 11 | rng.randrange(1 << 11) for _ in range(rng.randrange(1, 12))]
        rows = [[rng.randrange(1 << 16)] for _ in range(6)]
        prog = [0x17 << 11 | 1 << 8] + prog + [0x18 << 11 | 1 << 8, 0x01 << 11]
        outs = [rng.choice([0, r[0], 1]) for r in rows]
        whole = lib.evaluate(make_task("w", rows, outs), prog)
        each = sum(lib.evaluate(make_task("e", [r], [o]), prog) for r, o in zip(rows, outs))
        assert whole == each
        checked += whole > 0
    assert checked > 20
