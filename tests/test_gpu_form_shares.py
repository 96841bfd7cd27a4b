"""Rounds of few pairs of lists with many groups of terms (k_round_form): the lanes
that have no pair take groups, and a block takes fewer pairs. Row counts from one
pair up, two and three nodes (a zero in the eq point makes a round sum at a third),
with and without virtual tables, more and fewer groups than lanes, against the
oracle's restatement of gkr::prove_sumcheck (crates/gkr/src/lib.rs:792)."""
import random

import pytest

import oracle_lib as O
from test_gpu_gkr_sumcheck import _device, oracle_sumcheck

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


def circuit(cols, products, nv, virtuals):
    import circuits as C

    rng = random.Random(cols * 1000 + products)
    c = C.Circuit(nv, cols, virtuals)
    ops = [C.col(i) for i in range(cols)] + [C.virt(i) for i in range(len(virtuals))]
    coeff = lambda: rng.choice([1, C.P_R - 1, rng.randrange(2, C.P_R), rng.randrange(2, C.P_R)])  # noqa: E731
    gates = [C.quadratic(coeff(), [(coeff(), rng.choice(ops)) for _ in range(rng.randint(0, 2))],
                         [(coeff(), rng.choice(ops), rng.choice(ops)) for _ in range(6)])
             for _ in range((products + 5) // 6)]
    c.add_layer(gates[1:], enforcing=gates[:1])
    return c


@pytest.mark.parametrize("nv", [1, 2, 3, 4, 5, 6, 8, 10, 12])
@pytest.mark.parametrize("cols,products,virtuals", [(3, 6, ()), (24, 60, ()), (45, 400, ()), (45, 400, (0, 3)),
                                                    (120, 700, ()), (400, 900, (0,))])
def test_rounds_match_oracle(ctx, cols, products, virtuals, nv):
    import apogee_gpu as A

    if cols > 100 and nv > 8:
        pytest.skip("the oracle's time")
    rng = random.Random(nv)
    c = circuit(cols, products, nv, virtuals)
    blob = c.to_blob()
    n = len(c.layers[0][4]) + len(c.layers[0][5])
    weights = [rng.randrange(O.P_R) for _ in range(n)]
    point = [0 if j % 3 == 2 else rng.randrange(O.P_R) for j in range(nv)]
    lower = [[rng.choice([0, 1, rng.getrandbits(32), rng.randrange(O.P_R)]) for _ in range(1 << nv)]
             for _ in range(cols)]
    snap = A.transcript_append_scalars(A.transcript_init(), 41, [cols, nv])
    import torch

    dev = [_device(torch, t) for t in lower]
    got = ctx.gkr_prove_sumcheck(blob, 0, weights, {}, point, [t.data_ptr() for t in dev], None, snap)
    osnap = bytearray(snap)
    want = oracle_sumcheck(blob, 0, weights, {}, point, lower, [], osnap)
    assert got[0] == want[0] and got[1] == want[1] and got[2] == want[2] and got[3] == bytes(osnap)
