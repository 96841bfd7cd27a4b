"""Window tables of the resident SRS (over the stub runtime): how many points one
covers, and how long it lives once a larger one of its width replaces it."""
import pytest

import stub_runtime

pytestmark = pytest.mark.cpu_host

POINT = 64


def table_bytes(width, points):
    return (254 + 1 + width - 1) // width * points * POINT


@pytest.mark.parametrize("width,log_n", [(2, 13), (5, 13), (6, 16), (7, 16), (11, 16)])
def test_narrow_candidates_stay_within_a_prefix(width, log_n):
    """The autotuner times widths below 12 up to 2^16 points: it never needs their
    tables over more."""
    most, held = stub_runtime.run(f"""
ctx = A.Context(0)
ctx.srs_generate(5, 1 << 18)
ctx.commit(bytes(32 << 8), 8)
before = stub.held()
stub.reset()
ctx.msm_autotune(addr(bytes(32 << {log_n})), 1 << {log_n}, 8, {log_n}, cands=({width},))
result = [stub.most() - before, stub.held() - before]
""")
    scratch = 256 << 20  # buckets, sorted references and folds of a 2^16-point MSM
    assert most < 2 * table_bytes(width, 1 << 16) + scratch
    assert held < table_bytes(width, 1 << 16) + scratch
