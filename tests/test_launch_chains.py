"""A kernel launched with programmatic stream serialization waits, by its first
instruction, for the kernel before it on its stream. That wait is specified for
kernels, so such a launch may not come first after a copy, a memset, an event wait
or an allocation in stream order (nor first in a call, whose caller may have
queued any of these on the context's stream). Every entry point's host side runs
over the stub runtime, which notes what stands before each such launch."""
import pytest

import stub_runtime

pytestmark = pytest.mark.cpu_host

SETUP = """
class Ctx(A.Context):  # every call after work that the caller queued
    def __getattribute__(self, name):
        _lib.stub_caller()
        return super().__getattribute__(name)
ctx = Ctx(0)
ctx.srs_generate(5, 1 << LOG_SRS)
col = lambda nv: addr(bytes(32 << nv))
snap = A.transcript_append_scalars(A.transcript_init(), 7, [1, 2, 3])
inf = bytes(64)
rng = random.Random(1)
point = lambda n: [rng.randrange(A.P_R) for _ in range(n)]
"""

COMMITS = """
for nv in (2, 8, 12, 14):
    ctx.commit(bytes(32 << nv), nv)
    ctx.commit_device(col(nv), nv)
    ctx.commit_batch_device([col(nv)] * 3, nv)
    ctx.commit_batch([bytes(32 << nv)] * 3, nv)
    ctx.commit_u32([0] * (1 << nv), nv)
    for bits in (1, 8, 16, 32):
        ctx.commit_narrow(bytes(8 * ((max(1, bits) << nv) + 63)), bits, nv)
for k in (1, 2, 40):
    ctx.commit_stack([bytes(32 << 8)] * k, 8)
    ctx.commit_stack_device([col(8)] * k, 8)
ctx.commit_batch_device([col(16)] * 130, 16)  # two groups, two lanes
for n in (1, 40, 3000):
    ctx.msm(inf * n, bytes(32 * n))
    ctx.msm_small_u32(inf * n, [0] * n)
ctx.discharge_msms([0, 1] * 6, bytes(32 * 12), inf * 12, [12])
"""

OPENINGS = """
for nv in (2, 4, 8, 12, 14, 20, 22):
    ctx.open(bytes(32 << nv), nv, inf, point(nv), snap)
for nv, k in ((2, 1), (8, 3), (12, 40)):
    ctx.batch_open([col(nv)] * k, nv, [inf] * k, point(nv), snap, on_device=True)
    ctx.batch_open([bytes(32 << nv)] * k, nv, [inf] * k, point(nv), snap)
ctx.batch_open_stacked([[col(7)] * 2, [col(7)]], 7, [inf] * 2, point(7), point(1), snap, on_device=True)
ctx.batch_open_stacked([[bytes(32 << 7)] * 2, [bytes(32 << 7)]], 7, [inf] * 2, point(7), point(1), snap)
"""

SUMCHECKS = """
for nv in (0, 1, 2, 3, 5, 9, 13):
    for terms, k in (([(1, 0, 1)], 2), ([(1, 0, 1), (3, 2, None), (5, 1, 2)], 3)):
        ctx.prove_zerocheck(terms, [bytes(32 << nv)] * k, nv, snap)
        ctx.prove_zerocheck(terms, [col(nv)] * k, nv, snap, on_device=True)
        ctx.prove_zerocheck_narrow(terms, [addr(bytes(64 + (1 << nv)))] * k, [1, 8, 1][:k], nv, snap, on_device=True)
import shard
def prove(blob, ncols, nv, slots):
    ch = {s: 3 + s for s in slots}
    for base, dev in (([bytes(32 << nv)] * ncols, False), ([col(nv)] * ncols, True)):
        v = ctx.gkr_forward(blob, base, ch, on_device=dev)
        ctx.gkr_prove(blob, v, ch, snap)
        v.free()
    v = ctx.gkr_forward_narrow(blob, [addr(bytes(64 + (1 << nv)))] * ncols, [8] * ncols, ch, on_device=True)
    ctx.gkr_prove(blob, v, ch, snap)
    v.free()
for nv in (3, 8, 11):
    prove(shard.shard_circuit(nv, 4), 4, nv, [0])
    prove(C.shard_circuit(nv, 4).to_blob(), 4, nv, [0])
for seed in range(6):
    r = random.Random(seed)
    c = C.random_circuit(r, 6, 3, 4, [0, 2], slots=(0, 1))
    prove(c.to_blob(), 3, 6, [0, 1])
"""

SHARD = """
import shard
for nv in (8, 12):
    sh = A.Shard(shard.shard_circuit(nv, 5), [col(nv)] * 5, nv, 1, 2, 3, 0, 1 << nv)
    ctx.prove_shard(sh)
"""


CALLS = {"commits": (16, COMMITS), "openings": (22, OPENINGS), "sumchecks": (4, SUMCHECKS), "shard": (12, SHARD)}


@pytest.mark.parametrize("calls", list(CALLS))
def test_chained_launches_follow_kernels(calls):
    log_srs, script = CALLS[calls]
    launched, misplaced = stub_runtime.run(SETUP.replace("LOG_SRS", str(log_srs)) + "stub.reset()\n" + script +
                                           "result = [stub.launched(), stub.misplaced()]\n")
    assert sum(launched.values()) > 20
    assert misplaced == []
