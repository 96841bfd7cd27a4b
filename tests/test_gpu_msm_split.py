"""MSMs over the caller's bases, whose scalars are split into two halves of 127 bits
by the curve's endomorphism (up to 2^19 scalars): scalars at the edges of the split,
sizes at the edges of its windows, points at infinity, repeated and opposite, against
the oracle or the SRS's known tau."""
import random

import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
P = O.P_R
# lambda, and the short basis of {(x, y): x + lambda y = 0 mod r}.
LAM = 0xB3C4D79D41A917585BFC41088D8DAAA78B17EA66B99C90DD
A1, A2, B1 = 0x89D3256894D213E3, 0x6F4D8248EEB859FD0BE4E1541221250B, 0x6F4D8248EEB859FC8211BBEB7D4F1128
EDGES = sorted({(x + d) % P for x in (0, LAM, -LAM, LAM * LAM, A1, A2, B1, A1 * LAM, A2 * LAM, B1 * LAM, P // 2, P // 3,
                                      1 << 127, 1 << 128, 1 << 253, (1 << 127) * LAM, (A1 + A2) // 2,
                                      (A1 + A2) // 2 * LAM, (B1 - A1) // 2 * LAM, (A2 + B1) // 2 * (1 + LAM))
                for d in (-1, 0, 1)})


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


def test_basis():
    assert (LAM * LAM + LAM + 1) % P == 0
    assert (A1 - B1 * LAM) % P == 0 and (A2 + A1 * LAM) % P == 0 and A1 * A1 + A2 * B1 == P


def test_edge_scalars_one_at_a_time(ctx):
    import apogee_gpu as A

    p = O.g1_mul(O.G1_GEN, 0xABCDEF0123456789)
    for k in EDGES:
        assert ctx.msm(p, A.to_mont_bytes([k])) == O.g1_mul(p, k), hex(k)


@pytest.mark.parametrize("pattern", ["edges", "infinity", "opposite", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 2484])
def test_against_oracle(ctx, n, pattern):
    import apogee_gpu as A

    rng = random.Random(n)
    bases, scalars = O.msm_case("infinity" if pattern == "infinity" else "random", n, 90 + n)
    xs = [int.from_bytes(scalars[i:i + 32], "little") for i in range(0, len(scalars), 32)]
    if pattern == "edges":
        xs = [rng.choice(EDGES) for _ in xs]
    elif pattern == "mixed":
        xs = [rng.choice([0, 1, P - 1, rng.getrandbits(32), rng.getrandbits(127), x]) for x in xs]
    elif pattern == "opposite":  # P, -P, P, ... under one scalar: all or nothing remains
        x, y = bases[:32], int.from_bytes(bases[32:64], "little")
        q = O.P_Q
        bases = b"".join(x + (y if i % 2 == 0 else q - y).to_bytes(32, "little") for i in range(n))
        xs = [xs[0]] * n
    assert ctx.msm(bases, A.to_mont_bytes(xs)) == O.msm(bases, b"".join(O.fe(x) for x in xs), n, threads=8)


@pytest.mark.parametrize("n", [(1 << 14) - 1, 1 << 14, 1 << 16, (1 << 18) + 3, 1 << 19, (1 << 19) + 1])
def test_window_edges_known_tau(ctx, n):
    """The last two: the most scalars that are split, and one more."""
    import apogee_gpu as A

    tau = 0x5EED7654321
    if ctx.srs_len() < (1 << 19) + 1:
        ctx.srs_generate(tau, (1 << 19) + 1)
    rng = random.Random(n)
    pick = [rng.randrange(P) for _ in range(997)] + EDGES
    xs = [pick[(i * i + i // 7) % len(pick)] for i in range(n)]
    f, t = 0, 1
    for x in xs:
        f = (f + x * t) % P
        t = t * tau % P
    assert ctx.msm(ctx.srs_download(n), A.to_mont_bytes(xs)) == O.g1_mul(O.G1_GEN, f)


@pytest.mark.parametrize("at", [0, 300, 2483])
def test_refusals(ctx, at):
    import apogee_gpu as A

    bases, _ = O.msm_case("random", 2484, 3)
    mem = bytearray(A.to_mont_bytes([7] * 2484))
    mem[32 * at:32 * at + 32] = P.to_bytes(32, "little")
    with pytest.raises(A.ApogeeError) as e:
        ctx.msm(bases, bytes(mem))
    assert e.value.variant == "NonCanonical"
    good = A.to_mont_bytes([7] * 2484)
    off = bytearray(bases)
    off[64 * at] ^= 1
    with pytest.raises(A.ApogeeError):
        ctx.msm(bytes(off), good)
    assert ctx.msm(bases, good) == O.msm(bases, O.fe(7) * 2484, 2484, threads=8)
