"""The insert kernel's exact column ids: levels expanded with ids and without
them (an arena too small for their scratch) are the same and the oracle's, on
test counts at the edges of the flag planes and of the four-test words, with
one and two inputs: a wrong merge or a missed one shows in the survivors."""
import random

import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import OEP_EXACT, OEP_EXACT_LIVE, Engine, make_task

pytestmark = pytest.mark.gpu


def task(inputs, tests, seed):
    rng = random.Random(seed)
    rows = [[rng.choice([0, 1, 2, 0xFFFF, 0x8000, 0x7FFF, rng.randrange(1 << 16)])
             for _ in range(inputs)] for _ in range(tests)]
    return make_task("ids", rows, [rng.randrange(1 << 16) for _ in rows])


@pytest.mark.parametrize("mode", [OEP_EXACT, OEP_EXACT_LIVE])
@pytest.mark.parametrize("tests", [1, 2, 3, 4, 5, 15, 16, 17, 18, 31, 32])
def test_levels_same_with_and_without_ids(engine, tests, mode):
    from oracle import oracle as O
    for inputs in (1, 2):
        # level 2 fits this arena, the ids of its parents (a quarter of what
        # is free at most) do not
        arena = (48 if inputs == 1 else 74) if tests <= 16 else (64 if inputs == 1 else 96)
        small = Engine(0, arena << 20)
        try:
            t = task(inputs, tests, 100 * tests + inputs)
            want = engine.solve(t, max_depth=2, oep_mode=mode, count_levels=True)
            got = small.solve(t, max_depth=2, oep_mode=mode, count_levels=True)
        finally:
            small.close()
        assert got.level_survivors == want.level_survivors
        assert got.level_children == want.level_children
        assert (got.tried, got.pruned_cum) == (want.tried, want.pruned_cum)
        if mode == OEP_EXACT:
            r, _ = O.enumerate_task(t, 2, O.EXACT, 1 << 12)
            last = len(want.tried)
            assert want.tried == [r.tried[k] for k in range(last)]
            assert want.pruned_cum == [r.pruned_cum[k] for k in range(last)]
