"""An engine has what it needs from its creation: the largest batch of the
first solve takes no device memory, and answers as small ones do."""
import pytest

from pca_gb300.pcalib import Engine, device_memory, make_task

pytestmark = pytest.mark.gpu


def tasks(n):
    """Functions found at depths 0, 1 and 2, each with values of its own."""
    out = []
    for i in range(n):
        rows = [[(i * 31 + 7 * t + 3) & 0xFFFF] for t in range(5)]
        f = (lambda x: x, lambda x: 2 * x, lambda x: x * x + 1, lambda x: 0x3456)[i % 4]
        out.append(make_task(f"t{i}", rows, [f(r[0]) & 0xFFFF for r in rows]))
    return out


@pytest.mark.parametrize("n", [257, 8192])
def test_the_first_batch_is_the_largest(n):
    eng = Engine(0, 4 << 30)
    try:
        eng.solve_batch(tasks(4), max_depth=2, first_only=True, sol_cap=1)   # lazy loading
        before = device_memory(0)[0]
        got = eng.solve_batch(tasks(n), max_depth=2, first_only=True, sol_cap=1)
        assert device_memory(0)[0] >= before
        want = [eng.solve(t, max_depth=2, first_only=True, sol_cap=1) for t in tasks(8)]
        for i in list(range(8)) + list(range(n - 8, n)):
            assert got[i].optimal_depth == want[i % 4].optimal_depth
        assert [s.programs for s in got[:8]] == [s.programs for s in want]
    finally:
        eng.close()
