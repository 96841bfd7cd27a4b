"""Which kernels a gate list's sumcheck runs on, and what the choice costs the
host (over the stub runtime): a list is made a quadratic form only where that has
fewer products than the list and takes the host less than the interpreter would take
the device."""
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


@pytest.mark.parametrize("cols,gates,rows", [(32, 200, 4), (64, 500, 4), (200, 2000, 4), (200, 2000, 10)])
def test_products_of_cached_forms(cols, gates, rows):
    """(Multiplied out product by product, the first three took 0.04, 0.4 and 17 s.)"""
    t, _ = stub_runtime.run(PROVE + f"result = prove(cached_products({cols}, 8, {gates}, {rows}), {rows})")
    assert t < 0.25


@pytest.mark.parametrize("name", list(LISTS))
def test_interpreted_lists(name):
    kernels = stub_runtime.run(PROVE + f"""
import interpreter_lists
c = interpreter_lists.circuit({name!r})
result = prove(c, c.trace_vars)[1]
""")
    assert kernels == LISTS[name][-1]


@pytest.mark.parametrize("cols,forms,gates,rows", [(6, 2, 8, 8), (16, 4, 12, 4), (32, 8, 40, 4), (24, 8, 200, 2),
                                                   (32, 8, 200, 16)])
def test_cached_products_that_merge_keep_the_form(cols, forms, gates, rows):
    _, kernels = stub_runtime.run(PROVE + f"result = prove(cached_products({cols}, {forms}, {gates}, {rows}), {rows})")
    assert kernels == ["k_round_form"]


def test_long_plain_lists_keep_the_form():
    """24,000 products over 80 columns have 3,240 monomials."""
    t, kernels = stub_runtime.run(PROVE + "result = prove(plain_products(80, 2000, 12, 4), 4)")
    assert kernels == ["k_round_form"]
