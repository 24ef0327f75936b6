"""The costs an engine reports for the shape its deeper stages take."""
import pytest

from pca_gb300 import taskgen
from pca_gb300.pcalib import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth, split", [(4, 2), (5, 3), (4, 1), (5, 2)])
def test_the_lane_per_state_s_cost_is_reported(depth, split):
    s = depth - split
    eng = Engine(0, 16 << 30)
    try:
        before = eng.tuning()
        sol = eng.solve(taskgen.is_power2_task(1), max_depth=depth, split_depth=split, sol_cap=1)
        tun = eng.tuning()
    finally:
        eng.close()
    assert sol.optimal_depth == -1
    assert tun["chunk_choices"][s][3] == 1024
    # stages of more than 5e9 evaluations are timed
    if sol.evaluations[depth] > 5_000_000_000:
        assert tun["chunk_n"][s][3] > before["chunk_n"][s][3]
        assert 0 < tun["chunk_ms"][s][3] < 1e-9
    else:
        assert tun["chunk_n"][s][3] == before["chunk_n"][s][3]
    assert tun["chunk_n"][s][:3] == before["chunk_n"][s][:3]
    assert tun["first_tests_n"][s] == before["first_tests_n"][s]
