"""The staged round kernel of short quadratic forms at the shapes where it can
go wrong: one to many tables (pairs a block from 64 down to 1), linear and
repeated terms, fewer pairs than a block holds, one block and several, lists as
short as the rounds that end a proof; against the oracle, byte for byte."""
import random

import pytest

import oracle_lib as O
from test_gpu_zerocheck import run_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


def gate(rng, arity):
    terms = [(rng.choice([1, O.P_R - 1, rng.randrange(O.P_R)]), a, (a + 1) % arity) for a in range(arity)]
    terms += [(rng.randrange(O.P_R), rng.randrange(arity), None), (1, 0, 0), (O.P_R - 3, 0, None)]
    return terms


@pytest.mark.parametrize("arity", [1, 2, 3, 7, 40])
@pytest.mark.parametrize("nv", [0, 1, 2, 3, 4, 5, 6, 7, 9, 12])
def test_forms_match_oracle(ctx, arity, nv):
    if arity == 40 and nv > 9:
        pytest.skip("the oracle's time")
    rng = random.Random(1000 * arity + nv)
    cols = [[rng.choice([0, 1, rng.getrandbits(32), rng.randrange(O.P_R), O.P_R - 1]) for _ in range(1 << nv)]
            for _ in range(arity)]
    run_case(ctx, gate(rng, arity), cols, nv, 70 + nv)


@pytest.mark.parametrize("nv", [10, 16, 17])
def test_proof_of_many_blocks_verifies(ctx, nv):
    """2^16 pairs are more than one pass of the device: the proof of a gate that
    vanishes (a b - c) passes the verifier."""
    import apogee_gpu as A

    rng = random.Random(nv)
    a, b = ([rng.getrandbits(64) for _ in range(1 << nv)] for _ in range(2))
    terms, cols = [(1, 0, 1), (O.P_R - 1, 2, None)], [a, b, [x * y for x, y in zip(a, b)]]
    snap = A.transcript_init()
    rounds, finals, after = ctx.prove_zerocheck(terms, [A.to_mont_bytes(c) for c in cols], nv, snap)
    _, tr = A.verify_zerocheck(terms, 3, nv, rounds, finals, snap)
    assert tr == after
