"""Gate lists that no round kernel for quadratic forms takes (products of cached
linear forms over many columns: the form has more monomials than the list has
products), by name, with the interpreter kernels their sumcheck runs on, largest
rounds first: k_round, a thread a pair, or where there are few a thread a pair and
node; k_round_warp, a warp a pair, from sixteen gates on and wherever a round is
small."""
import random

import circuits as C

# name: (columns, cached forms, gates, enforcing gates among them, log2 of the rows,
# virtual tables, kernels)
LISTS = {
    "thread a pair": (24, 2, 15, 1, 17, (), ["k_round", "k_round_warp"]),
    "thread a pair and node": (40, 3, 15, 2, 13, (), ["k_round", "k_round_warp"]),
    "sixteen threads a block": (130, 4, 3, 0, 13, (), ["k_round", "k_round_warp"]),
    "eight threads a block": (200, 8, 2, 1, 13, (), ["k_round", "k_round_warp"]),
    "with virtual tables": (40, 3, 15, 1, 13, (C.V_ROW, C.V_RANGE16), ["k_round", "k_round_warp"]),
    "warp a pair": (60, 3, 40, 3, 13, (), ["k_round_warp"]),
    "warp a pair, virtual tables": (40, 2, 17, 0, 13, (C.V_ROW,), ["k_round_warp"]),
    "one row": (60, 2, 16, 1, 0, (), []),
    "two rows": (60, 2, 3, 1, 1, (), ["k_round_warp"]),
    "small, few gates": (60, 2, 3, 0, 5, (), ["k_round_warp"]),
    "small, many gates": (80, 2, 33, 2, 5, (C.V_ROW,), ["k_round_warp"]),
}


def circuit(name):
    cols, forms, gates, enforcing, nv, virtuals, _ = LISTS[name]
    rng = random.Random(name)
    c = C.Circuit(nv, cols, virtuals)
    ops = [C.col(i) for i in range(cols)] + [C.virt(i) for i in range(len(virtuals))]
    cached = [C.linear([(rng.randrange(2, C.P_R), o) for o in ops], rng.randrange(C.P_R)) for _ in range(forms)]
    pick = lambda: C.cached(rng.randrange(forms))  # noqa: E731
    made = []
    for j in range(gates):
        if j % 3 == 0:
            made.append(C.product(rng.randrange(2, C.P_R), pick(), pick()))
        elif j % 3 == 1:
            made.append(C.mask(pick(), pick()))
        else:
            made.append(C.quadratic(("ch", 0), [(1, rng.choice(ops))], [(C.P_R - 1, pick(), pick()),
                                                                        (("ch", 0), pick(), rng.choice(ops))]))
    n = gates - enforcing
    c.add_layer(made[:n], cached=cached, enforcing=made[n:])
    return c
