"""A solve leaves nothing of itself on the device when it returns: its arena
may be another stream's next (a server's slices), and what a task solved
before the search (its input is its output) has put there would land in it."""
import pytest
import torch

from pca_gb300 import taskgen
from pca_gb300.pcalib import make_task

pytestmark = pytest.mark.gpu


def identity(inputs, tests, seed):
    rows = [[(seed * 7919 + 31 * t + i) & 0xFFFF for i in range(inputs)] for t in range(tests)]
    return make_task("same", rows, [r[0] for r in rows])


def stream_of(engine):
    return torch.cuda.ExternalStream(engine.lib.pcagb_engine_stream(engine.h))


@pytest.mark.parametrize("tests", [1, 16, 17, 32])
@pytest.mark.parametrize("max_depth", [0, 1, 5])
def test_a_task_solved_at_depth_0_launches_nothing(engine, tests, max_depth):
    st = stream_of(engine)
    for task, depth in ((identity(1, tests, 3), 0),
                        (make_task("none", [[2 * t + 1] for t in range(tests)], [0] * tests), -1)):
        if depth < 0 and max_depth:
            continue
        for many in (False, True):
            if many:
                s = engine.solve_batch([task] * 300, max_depth=max_depth, first_only=True)[299]
            else:
                s = engine.solve(task, max_depth=max_depth)
            assert st.query()
            assert s.optimal_depth == depth
            assert s.kernel_launches == 0 and s.h2d_bytes == 0


def test_a_batch_of_both_kinds(engine):
    """Tasks solved at depth 0 among others, and levels kept for a caller
    that reads them (counters) even where no depth is searched."""
    st = stream_of(engine)
    rest = [t for _, t in taskgen.poisson_stream(6, rate=100.0, seed=21)]
    mix = [identity(2, 9, 1), *rest, identity(1, 32, 2)]
    got = engine.solve_batch(mix, max_depth=3, first_only=True, sol_cap=4)
    assert st.query()
    for t, s in zip(mix, got):
        alone = engine.solve(t, max_depth=3, first_only=True, sol_cap=4)
        assert (s.optimal_depth, s.programs[:1]) == (alone.optimal_depth, alone.programs[:1])
    s = engine.solve(mix[0], max_depth=3, count_levels=True)
    assert st.query() and s.optimal_depth == 0 and s.programs


def test_a_slice_given_back_is_written_by_its_next_solve_only(engine):
    """Requests solved at depth 0 and others in turn on a pool of two slices:
    each answer is the task's alone."""
    from pca_gb300.serve import NativeServer
    rest = [t for _, t in taskgen.poisson_stream(40, rate=100.0, seed=5)]
    alone = [engine.solve(t, max_depth=3, sol_cap=16, first_only=True) for t in rest]
    srv = NativeServer(workers=4, max_batch=1, max_depth=3, pool_bytes=2 * (64 << 20),
                       arena_bytes=64 << 20)
    try:
        for turn in range(3):
            reqs = []
            for i, t in enumerate(rest):
                for k in range(3):
                    # depth limits of 5 lay out more than the others'
                    reqs.append((srv.submit(0, identity(1 + k % 2, 32, i + k), max_depth=5), None))
                reqs.append((srv.submit(0, t), alone[i]))
            for r, want in reqs:
                assert r.done.wait(120) and r.error is None
                if want is None:
                    assert r.solution.optimal_depth == 0
                else:
                    assert (r.solution.optimal_depth, r.solution.programs) == (want.optimal_depth,
                                                                               want.programs)
    finally:
        srv.close()
