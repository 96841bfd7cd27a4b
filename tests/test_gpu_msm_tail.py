"""The edge-run folds and the bucket reduction at the sizes where their levels
change: one fold block against several (252 items, 2 a segment of 4 digits),
two items a quad against four (15,876), reductions of one block and of two
levels; against the oracle or the SRS's known tau."""
import random

import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


# 29 windows of 9 bits, 4 digits a segment: 126 segments at 17 points (5-bit
# windows below 2^9 points: fewer), 7,938 at 1,095.
@pytest.mark.parametrize("kind", ["random", "one_digit", "two_runs"])
@pytest.mark.parametrize("n", [1, 9, 10, 17, 18, 71, 1094, 1095, 1096, 8900])
def test_fold_levels_against_oracle(ctx, n, kind):
    import apogee_gpu as A

    bases, scalars = O.msm_case("random", n, 40 + n)
    if kind == "one_digit":  # every window one run over the whole list
        k = sum(5 << (9 * w) for w in range(27))
        scalars = O.fe(k) * n
    elif kind == "two_runs":
        a, b = sum(3 << (9 * w) for w in range(27)), sum(4 << (9 * w) for w in range(27))
        scalars = O.fe(a) * (n // 3) + O.fe(b) * (n - n // 3)
    xs = [int.from_bytes(scalars[i:i + 32], "little") for i in range(0, len(scalars), 32)]
    assert ctx.msm(bases, A.to_mont_bytes(xs)) == O.msm(bases, scalars, n, threads=8)


@pytest.mark.parametrize("cbits", [2, 4, 8, 9, 10, 12, 15, 17, 19])
def test_reduction_widths_known_tau(ctx, cbits):
    """K = 2^(cbits - 1) buckets: up to 256 in one block, more in two levels."""
    import torch

    import apogee_gpu as A

    tau, nv = 0x5EED1234567, 10
    n = 1 << nv
    ctx.srs_generate(tau, n)
    rng = random.Random(cbits)
    xs = [rng.choice([0, 1, rng.getrandbits(32), rng.randrange(O.P_R), O.P_R - 1]) for _ in range(n)]
    mem = A.to_mont_bytes(xs)
    d = torch.frombuffer(bytearray(mem), dtype=torch.uint8).cuda()
    assert ctx.msm_autotune(d.data_ptr(), n, nv, nv, cands=(cbits,)) == {nv: cbits}
    f_tau = sum(c * pow(tau, i, O.P_R) for i, c in enumerate(xs)) % O.P_R
    assert ctx.commit(mem, nv) == O.g1_mul(O.G1_GEN, f_tau)
    assert ctx.commit_batch_device([d.data_ptr()] * 3, nv) == [O.g1_mul(O.G1_GEN, f_tau)] * 3


@pytest.mark.parametrize("bits", [1, 8, 16, 32])
@pytest.mark.parametrize("nv", [2, 8, 12, 14, 18])
def test_few_bucket_digits_known_tau(ctx, nv, bits):
    """Narrow columns, whose digits fill few buckets: one scalar a thread, a
    ragged tile, several tiles a block; random values and all of the largest."""
    import apogee_gpu as A

    tau, n, p = 0xA5A5A5A5A5, 1 << nv, O.P_R
    if ctx.srs_len() != 1 << 18:
        ctx.srs_generate(tau, 1 << 18)
    rng = random.Random(100 * nv + bits)
    for vals in ([rng.getrandbits(bits) for _ in range(n)], [(1 << bits) - 1] * n):
        f_tau, x = 0, 1
        for v in vals:
            f_tau, x = (f_tau + v * x) % p, x * tau % p
        assert ctx.commit_narrow(A.narrow_bytes(vals, bits), bits, nv) == O.g1_mul(O.G1_GEN, f_tau)


@pytest.mark.parametrize("kind", ["uniform", "equal"])
def test_pair_rounds_degenerate_bases(ctx, kind):
    """2^20 generic bases drawn from {infinity, G, -G, 2G, 3G, 7G}: 17 windows,
    above the affine pair rounds' least size, so adjacent points of a bucket
    collide in every way the rounds classify. The value is (sum s_i k_i) G."""
    import apogee_gpu as A

    rng = random.Random(13)
    n = 1 << 20
    ks = [0, 1, O.P_R - 1, 2, 3, 7]
    pts = {k: (bytes(64) if k == 0 else O.g1_mul(O.G1_GEN, k)) for k in ks}
    kk = rng.choices(ks, k=n)
    ss = [rng.randrange(O.P_R)] * n if kind == "equal" else [rng.randrange(O.P_R) for _ in range(n)]
    want = O.g1_mul(O.G1_GEN, sum(s * k for s, k in zip(ss, kk)) % O.P_R)
    assert ctx.msm(b"".join(pts[k] for k in kk), A.to_mont_bytes(ss)) == want
