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


def test_a_replaced_table_is_freed():
    small, large = stub_runtime.run("""
ctx = A.Context(0)
ctx.srs_generate(5, 1 << 19)
data = [addr(bytes(32 << 14))] * 3
ctx.commit_batch_device(data, 14)
before = stub.held()
ctx.srs_prepare(13)
result = [before, stub.held()]
""")
    assert large - small == table_bytes(13, 1 << 19) - table_bytes(13, 1 << 18)


def test_a_replaced_table_lives_while_another_context_reads_it():
    held = stub_runtime.run("""
ctx = A.Context(0)
ctx.srs_generate(5, 1 << 19)
data = [addr(bytes(32 << 14))] * 3
ctx.commit_batch_device(data, 14)
result = [stub.held()]
other = A.Context(0)
other.srs_share(ctx)
base = stub.held()
ctx.srs_prepare(13)
result.append(stub.held() - base)
other.commit_batch_device(data, 14)  # the table it borrowed: none is built
result.append(stub.launched().get("k_window_table", 0))
other.srs_share(ctx)
before = stub.held()
other.commit_batch_device(data, 14)
result.append(stub.held() - before)
del other
import gc
gc.collect()
result.append(stub.held())
""")
    old, new = table_bytes(13, 1 << 18), table_bytes(13, 1 << 19)
    assert held[1] == new
    assert held[2] == 2
    assert held[3] == 0
    assert held[4] == held[0] + new - old
