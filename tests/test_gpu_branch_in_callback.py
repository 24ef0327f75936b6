"""Branch mode called while a solve of the same engine runs (from the solve's
own callbacks, from another thread): both answers are those of the calls
alone, because the search takes the engine's arena only where no solve uses
it."""
import random
import threading

import pytest
import torch

from pca_gb300 import taskgen
from pca_gb300.pcalib import Engine, make_task

pytestmark = pytest.mark.gpu
M = 0xFFFF


def branch_task(seed, f=lambda x: 0 if x & 0x8000 else x, tests=11):
    rng = random.Random(seed)
    rows = [[v] for v in (0, 1, M, 0x7FFF, 0x8000)]
    rows += [[rng.randrange(1 << 16)] for _ in range(tests - len(rows))]
    return make_task("branch", rows, [f(r[0]) for r in rows])


def branch_answer(s):
    return (s.optimal_depth, s.total_solutions, s.programs, s.tried, s.pruned_cum)


def answer(s):
    return (s.optimal_depth, s.total_solutions, s.programs, s.candidates)


@pytest.fixture(scope="module")
def eng():
    e = Engine(0, 8 << 30)
    yield e
    e.close()


@pytest.mark.parametrize("depth", [2, 3])
def test_in_an_order_callback(eng, depth):
    bt = branch_task(1)
    want = branch_answer(eng.solve_branch(bt, max_depth=depth))
    task = taskgen.is_power2_task(1)
    found = make_task("mix", [[1], [2], [7], [9]], [14, 28, 98, 126])
    for t in (task, found):
        calls = []

        def order(view, branch):
            out = torch.arange(view.n - 1, -1, -1, device="cuda", dtype=torch.int32)
            torch.cuda.synchronize()
            if branch:
                calls.append(branch_answer(eng.solve_branch(bt, max_depth=depth)))
            return out

        run = lambda branch: answer(eng.solve_ordered(  # noqa: E731
            t, lambda v: order(v, branch), chunk=1 << 20, max_depth=3, split_depth=2))
        alone = run(False)
        assert run(True) == alone
        assert calls and all(c == want for c in calls)
    # given back: the search has it again, and then the solve
    assert branch_answer(eng.solve_branch(bt, max_depth=depth)) == want


def test_in_a_batch_s_delivery(eng):
    bt = branch_task(2)
    want = branch_answer(eng.solve_branch(bt, max_depth=2))
    tasks = [t for _, t in taskgen.poisson_stream(8, rate=100.0, seed=21)]
    alone = [answer(s) for s in eng.solve_batch(tasks, max_depth=3, sol_cap=4)]
    seen = []
    got = eng.solve_batch(tasks, max_depth=3, sol_cap=4, on_done=lambda i, s: seen.append(
        branch_answer(eng.solve_branch(bt, max_depth=2))))
    assert [answer(s) for s in got] == alone
    assert len(seen) == len(tasks) and all(s == want for s in seen)


def test_from_another_thread(eng):
    """A search in one thread and solves in another: whichever comes first
    has the arena, the search does without it or the solve waits for it."""
    bt, task = branch_task(3), taskgen.is_power2_task(2)
    want_b = branch_answer(eng.solve_branch(bt, max_depth=2))
    want_s = answer(eng.solve(task, max_depth=3, split_depth=2))
    got, errors = [], []

    def search():
        try:
            for _ in range(30):
                got.append(branch_answer(eng.solve_branch(bt, max_depth=2)))
        except Exception as exc:  # noqa: BLE001
            errors.append(exc)

    th = threading.Thread(target=search)
    th.start()
    for _ in range(60):
        assert answer(eng.solve(task, max_depth=3, split_depth=2)) == want_s
    th.join(60)
    assert not th.is_alive() and not errors
    assert got == [want_b] * 30
