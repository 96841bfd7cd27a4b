"""Layers of many hundred columns: row-wise lists whose pair's values nearly fill a
block's shared memory, halving lists of twice as many tables, and the forward pass
over both, against the oracle. (Lists of more than 2,132 tables are refused.)"""
import pytest

from test_gpu_gkr import run_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


def wide(cols, nv):
    import circuits as C

    c = C.Circuit(nv, cols)
    c.add_layer([C.product(2 + j, C.col(j), C.col((j + 1) % cols)) for j in range(cols)],
                enforcing=[C.linear([(1 + j, C.col(j)) for j in range(cols)], 3)])
    c.add_layer([C.tree_product(C.col(j)) if j % 3 else C.tree_cross(C.col(j), C.col((j + 5) % cols))
                 for j in range(cols)], halving=True)
    return c


@pytest.mark.parametrize("cols,nv", [(420, 1), (420, 6), (700, 3), (1060, 1), (1060, 4)])
def test_wide_layers_match_oracle(ctx, cols, nv):
    run_case(ctx, wide(cols, nv), cols + nv)


def test_wider_lists_are_refused(ctx):
    import apogee_gpu as A

    cols = 2200
    blob = wide(cols, 3).to_blob()
    ch = {s: 1 + s for s in (0, 1, 2)}
    with pytest.raises(A.ApogeeError) as e:
        v = ctx.gkr_forward(blob, [A.to_mont_bytes([j] * 8) for j in range(cols)], ch)
        ctx.gkr_prove(blob, v, ch, A.transcript_init())
    assert e.value.variant == "BadCircuit"
