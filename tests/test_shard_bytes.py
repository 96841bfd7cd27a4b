"""apg_shard_device_bytes against what proving the shard takes (over the stub
runtime): the server admits requests by it, so it is at least the real peak, and no
more than a quarter and the buffers' fixed part above it."""
import pytest

import stub_runtime

pytestmark = pytest.mark.cpu_host

PROVE = """
import shard
ctx = A.Context(0)
ctx.srs_generate(5, 1 << max(nv, 8))
ctx.srs_prepare()
cols = [addr(bytes(32 << nv))] * k
sh = A.Shard(shard.shard_circuit(nv, k), cols, nv, 1, 2, 3, 0, 1 << nv)
A.lib().apg_shard_device_bytes.restype = ctypes.c_size_t
need = A.lib().apg_shard_device_bytes(ctypes.byref(sh.c))
before = stub.held()
stub.reset()
ctx.prove_shard(sh)
result = [need, stub.most() - before]
"""


# One group a commit and two lanes of two, three and four; every default window
# width; with and without the pair rounds' lists (from 2^24 digits; an opening's
# from 2^23), and lists at their largest.
@pytest.mark.parametrize("nv,k", [(8, 1), (8, 4), (8, 16), (10, 16), (12, 4), (12, 16), (14, 2), (14, 16), (14, 40),
                                  (16, 1), (16, 12), (16, 16), (18, 4), (18, 16), (18, 40), (20, 4), (20, 16)])
def test_estimate_covers_the_peak(nv, k):
    need, peak = stub_runtime.run(f"nv, k = {nv}, {k}\n" + PROVE)
    assert peak <= need <= peak + peak // 4 + (64 << 20)
