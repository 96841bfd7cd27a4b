"""Openings at the sizes where the opening's passes change shape: transforms of
4 to 4096 points in one block and above, suffix scans of one block a column and
segmented ones, dots of one and of several reductions, more columns than a
reduction takes. Each passes the deferred verifier under the SRS's tau, values
included (they are part of the claim)."""
import random

import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
TAU = 0x5151515151


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        c.srs_generate(TAU, 1 << 24)
        yield c


@pytest.mark.parametrize("nv,k", [(2, 1), (4, 17), (8, 31), (14, 2), (16, 3), (18, 16), (20, 1), (22, 1), (24, 1)])
def test_openings_verify(ctx, nv, k):
    import torch

    import apogee_gpu as A
    import synth

    rng = random.Random(nv)
    n = 1 << nv
    cols = [synth.device_column(ctx, torch, n, 900 + 40 * nv + j, "mixed" if j else "uniform") for j in range(k)]
    for t in cols:
        ctx.fr_to_mont_device(t.data_ptr(), n)
    ptrs = [t.data_ptr() for t in cols]
    cms = ctx.commit_batch_device(ptrs, nv)
    u = [rng.randrange(O.P_R) for _ in range(nv)]
    snap = A.transcript_append_scalars(A.transcript_init(), 39, [nv, k])
    vs, proof, after = ctx.batch_open(ptrs, nv, cms, u, snap, on_device=True)
    sides, scalars, points, tr = A.mercury_batch_verify_deferred(cms, u, vs, proof, snap)
    assert tr == after
    rc, a, b, _, _ = O.accumulator_msms(sides, scalars, points, [12], weights=[1])
    assert rc == 0 and a == O.g1_mul(b, TAU)
