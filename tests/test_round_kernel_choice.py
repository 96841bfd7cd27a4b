"""Which kernels a gate list's sumcheck runs on, and what the choice costs the
host (over the stub runtime): a list is expanded to a quadratic form only where
the expansion is small against the list or against its rounds, whatever its gates'
operands; beyond that the interpreter takes it as it stands."""
import pytest

import stub_runtime
from interpreter_lists import LISTS

pytestmark = pytest.mark.cpu_host

PROVE = """
ctx = A.Context(0)
def prove(c, nv):
    width = c.n_committed
    n = len(c.layers[0][4]) + len(c.layers[0][5])
    tables = [addr(bytes(32 << nv)) for _ in range(width)]
    blob, weights, point = c.to_blob(), list(range(2, 2 + n)), list(range(3, 3 + nv))
    snap = A.transcript_init()
    stub.reset()
    t = time.perf_counter()
    ctx.gkr_prove_sumcheck(blob, 0, weights, {0: 7}, point, tables, None, snap)
    t = time.perf_counter() - t
    return t, sorted(k for k in stub.launched() if k.startswith("k_round"))
def cached_products(cols, forms, gates, nv):
    r = random.Random(cols)
    c = C.Circuit(nv, cols)
    cac = [C.linear([(r.randrange(2, A.P_R), C.col(i)) for i in range(cols)], 3) for _ in range(forms)]
    c.add_layer([C.product(5, C.cached(r.randrange(forms)), C.cached(r.randrange(forms))) for _ in range(gates)],
                cached=cac)
    return c
def plain_products(cols, gates, terms, nv):
    r = random.Random(cols)
    c = C.Circuit(nv, cols)
    c.add_layer([C.quadratic(1, [], [(r.randrange(2, A.P_R), C.col(r.randrange(cols)), C.col(r.randrange(cols)))
                                     for _ in range(terms)]) for _ in range(gates)])
    return c
"""


@pytest.mark.parametrize("cols,gates", [(32, 200), (64, 500), (200, 2000)])
def test_products_of_cached_forms_are_not_multiplied_out(cols, gates):
    t, kernels = stub_runtime.run(PROVE + f"result = prove(cached_products({cols}, 8, {gates}, 4), 4)")
    assert kernels == ["k_round_warp"]
    # (multiplied out, the three took 0.04, 0.4 and 17 s; parsing the blob and
    # packing the gates takes milliseconds)
    assert t < 0.25


@pytest.mark.parametrize("name", list(LISTS))
def test_interpreted_lists(name):
    kernels = stub_runtime.run(PROVE + f"""
import interpreter_lists
c = interpreter_lists.circuit({name!r})
result = prove(c, c.trace_vars)[1]
""")
    assert kernels == LISTS[name][-1]


def test_small_cached_products_keep_the_form():
    _, kernels = stub_runtime.run(PROVE + "result = prove(cached_products(6, 2, 8, 8), 8)")
    assert kernels == ["k_round_form"]


def test_long_plain_lists_keep_the_form():
    """24,000 products over 80 columns have 3,240 monomials."""
    t, kernels = stub_runtime.run(PROVE + "result = prove(plain_products(80, 2000, 12, 4), 4)")
    assert kernels == ["k_round_form"]
