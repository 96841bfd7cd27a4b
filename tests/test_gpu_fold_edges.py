"""The edge-run folds where their levels change. A call of E possible digits makes
2 ceil(E / s) items, s = 4 up to 2^15 digits and 8 above: one block folds up to 504
items, two items a quad up to 31,752, four above; more slices than the device holds
at once are made longer. Over the caller's bases n scalars are 2n halves of 16
windows of 8 bits (up to 2^15 halves), E = 32 n; over the SRS's tables a column of
n <= 2^8 points has 43 n digits. Against the oracle or the SRS's known tau."""
import random

import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
# lambda (the scalars' endomorphism): k1 + lambda k2 splits into (k1, k2), both well
# below 2^125 here.
LAM = 0xB3C4D79D41A917585BFC41088D8DAAA78B17EA66B99C90DD


def items(e):
    s = 4 if e <= 1 << 15 else 8
    return 2 * -(-e // s)


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


def test_the_sizes_are_the_edges():
    assert [items(32 * n) for n in (31, 32)] == [496, 512]
    assert [items(32 * n) for n in (3968, 3969, 3970)] == [31744, 31752, 31760]
    assert [items(43 * 4 * k) for k in (5, 6)] == [430, 516]
    assert [items(43 * 256 * k) for k in (11, 12)] == [30272, 33024]
    assert items(32 * 1024) == 16384 and items(32 * 1025) == 8200


@pytest.mark.parametrize("kind", ["random", "one_digit", "two_runs", "few_digits"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 3968, 3969, 3970])
def test_caller_bases_against_oracle(ctx, n, kind):
    import apogee_gpu as A

    def all_windows(d):  # digit d in every window but the top one of both halves
        k = sum(d << (8 * w) for w in range(15))
        return (k + LAM * k) % O.P_R

    bases, scalars = O.msm_case("random", n, 70 + n)
    rng = random.Random(n)
    xs = [int.from_bytes(scalars[i:i + 32], "little") for i in range(0, len(scalars), 32)]
    if kind == "one_digit":  # every window one run over the whole list
        xs = [all_windows(5)] * n
    elif kind == "two_runs":
        xs = [all_windows(3)] * (n // 3) + [all_windows(4)] * (n - n // 3)
    elif kind == "few_digits":  # runs that end anywhere in a block
        xs = [all_windows(rng.choice([1, 2, 60])) if rng.random() < 0.9 else rng.choice([0, 1, x]) for x in xs]
    want = O.msm(bases, b"".join(O.fe(x) for x in xs), n, threads=8)
    assert ctx.msm(bases, A.to_mont_bytes(xs)) == want


@pytest.mark.parametrize("kind", ["uniform", "bits", "one_value"])
@pytest.mark.parametrize("nv,k", [(2, 1), (2, 5), (2, 6), (8, 2), (8, 3), (8, 11), (8, 12)])
def test_commits_known_tau(ctx, nv, k, kind):
    import torch

    import apogee_gpu as A

    tau, n, p = 0xC0FFEE123457, 1 << nv, O.P_R
    if ctx.srs_len() != 1 << 8:
        ctx.srs_generate(tau, 1 << 8)
    rng = random.Random(100 * nv + k)
    one = rng.randrange(p)
    draw = {"uniform": lambda: rng.randrange(p), "bits": lambda: rng.getrandbits(1), "one_value": lambda: one}[kind]
    cols = [[draw() for _ in range(n)] for _ in range(k)]
    dev = [torch.frombuffer(bytearray(A.to_mont_bytes(c)), dtype=torch.uint8).cuda() for c in cols]
    want = [O.g1_mul(O.G1_GEN, sum(c * pow(tau, i, p) for i, c in enumerate(col)) % p) for col in cols]
    assert ctx.commit_batch_device([d.data_ptr() for d in dev], nv) == want
