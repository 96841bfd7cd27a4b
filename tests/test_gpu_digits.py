"""The digit passes over many buckets (17-bit windows, from 2^18 rows): scalars whose
digits lie in the low windows only, in the upper ones only, at a digit's or a carry's
edge, all in one bucket, in a few, or in as many as there are lanes, at lengths that
end inside a warp or a block; commitments against the SRS's known tau."""
import random

import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
P = O.P_R
TAU, LOG = 0x5EED0123, 18


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        c.srs_generate(TAU, 1 << LOG)
        c.srs_prepare(17)
        yield c


def _pool(kind, rng):
    edge = [(1 << 17) - 1, 1 << 16, (1 << 16) - 1, (1 << 16) + 1, (1 << 33) - 1, (1 << 34) - 1, 1 << 34, 1 << 32,
            (1 << 32) - 1, (1 << 64) - 1, 1 << 64, P - 1, P - 2, sum((1 << 16) << (17 * w) for w in range(14)),
            sum(((1 << 17) - 1) << (17 * w) for w in range(14)) % P]
    return {"zero": [0], "bits": [0, 1], "u32": [rng.getrandbits(32) for _ in range(4096)], "edge": edge,
            "one_value": [rng.randrange(P)], "few": [rng.randrange(P) for _ in range(3)],
            "lanes": [rng.randrange(P) for _ in range(37)],
            "upper": [rng.getrandbits(200) << 51 for _ in range(997)],
            "sparse": [0] * 200 + [rng.randrange(P), 1, (1 << 34) - 1],
            "random": [rng.randrange(P) for _ in range(4099)]}[kind]


@pytest.mark.parametrize("kind", ["zero", "bits", "u32", "edge", "one_value", "few", "lanes", "upper", "sparse",
                                  "random"])
def test_commitments_known_tau(ctx, kind):
    import torch

    import apogee_gpu as A

    rng = random.Random(kind)
    pool = [x % P for x in _pool(kind, rng)]
    n = 1 << LOG
    at = [(i * i + i // 5) % len(pool) for i in range(n)]
    mont = [A.to_mont_bytes([x]) for x in pool]
    d = torch.frombuffer(bytearray(b"".join(mont[k] for k in at)), dtype=torch.uint8).cuda()
    torch.cuda.synchronize()
    f, t = 0, 1
    for k in at:
        f = (f + pool[k] * t) % P
        t = t * TAU % P
    want = O.g1_mul(O.G1_GEN, f)
    assert ctx.commit_device(d.data_ptr(), LOG) == want
    assert ctx.commit_batch_device([d.data_ptr()] * 2, LOG) == [want] * 2


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 300])
def test_odd_lengths_with_wide_windows(ctx, n):
    """Openings commit to vectors of any length; a generic MSM of 12-bit windows runs
    the same kernel (2^15 half scalars and more)."""
    import apogee_gpu as A

    m = (1 << 14) + n
    rng = random.Random(n)
    pool = [rng.randrange(P) for _ in range(61)] + [0, 1, P - 1, 1 << 40]
    xs = [pool[(i * i + 3 * i) % len(pool)] for i in range(m)]
    f, t = 0, 1
    for x in xs:
        f = (f + x * t) % P
        t = t * TAU % P
    assert ctx.msm(ctx.srs_download(m), A.to_mont_bytes(xs)) == O.g1_mul(O.G1_GEN, f)
