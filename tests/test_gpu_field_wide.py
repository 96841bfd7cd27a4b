"""Sums of up to fifteen products with one reduction, against integers: the
largest operands at every count (the sum next to 2^512, its reduced value past
twice the modulus), carries between the halves, and sums whose reduced value,
before the last subtractions, lies just below and just above m, 2m and 3m."""
import os
import random
import subprocess

import pytest

import apogee_gpu as A
from test_gpu_field import edge_values

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
R = 1 << 256
MOST = 15


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "field_wide_check")
    import build_lib

    subprocess.check_call([build_lib._nvcc()] + build_lib.ARCH +
                          ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-o", exe,
                           os.path.join(HERE, "native", "field_wide_check.cu")])
    return exe


def before_subtraction(total, p):
    """(T + M p) / R with the M below R that clears T's low half."""
    return (total + (-total * pow(p, -1, R)) % R * p) // R


def near(target, p, rng):
    """Fifteen products at most whose sum's high part puts the reduced value within
    2^140 or so of `target`, from either side."""
    sums = []
    for _ in range(200):
        goal = target + rng.randrange(-(1 << 140), 1 << 140)
        # (T + M p) / R is about T / R + (M / R) p, M as good as random: steer with T
        # = goal R - M p for a chosen M, its low half then fixed by M.
        M = rng.randrange(R)
        total = goal * R - M * p
        if total <= 0 or total >= MOST * (p - 1) ** 2:
            continue
        pairs, left = [], total
        while left > 0 and len(pairs) < MOST - 2:
            a = p - 1 - rng.randrange(1 << 64)
            b = min(left // a, p - 1)
            if b == 0:
                break
            pairs.append((a, b))
            left -= a * b
        if left < p:  # what remains, a multiple of one
            if left:
                pairs.append((left, 1))
        elif left < (p - 1) ** 2:
            b = p - 1
            pairs += [(left // b, b)] + ([(left % b, 1)] if left % b else [])
        else:
            continue
        if len(pairs) <= MOST and all(0 <= x < p for q in pairs for x in q):
            assert sum(a * b for a, b in pairs) == total
            sums.append(pairs)
    return sums


def cases(p):
    rng = random.Random(11)
    edge = edge_values(p, rng)
    out = [[(p - 1, p - 1)] * k for k in range(MOST + 1)]
    out += [[(v, p - 1)] * k for v in edge for k in (1, 2, 14, MOST)]
    out += [[(v, v)] * k for v in edge for k in (2, 7, MOST)]
    out += [[(rng.choice(edge), rng.choice(edge)) for _ in range(k)] for k in range(1, MOST + 1) for _ in range(40)]
    out += [[(rng.randrange(p), rng.randrange(p)) for _ in range(k)] for k in range(1, MOST + 1) for _ in range(20)]
    for m in (1, 2, 3):
        out += near(m * p, p, rng)
    return out


@pytest.mark.parametrize("p", [A.P_Q, A.P_R])
def test_the_cases_reach_the_edges(p):
    seen = [before_subtraction(sum(a * b for a, b in c), p) for c in cases(p)]
    assert max(seen) < 4 * p and max(seen) > 3 * p
    for m in (1, 2, 3):
        assert any(-(1 << 200) < v - m * p < 0 for v in seen) and any(0 <= v - m * p < 1 << 200 for v in seen)
    assert max(sum(a * b for a, b in c) for c in cases(p)) == MOST * (p - 1) ** 2 < 1 << 512


@pytest.mark.parametrize("field,p", [("q", A.P_Q), ("r", A.P_R)])
def test_sums_of_products(checker, field, p):
    sums = cases(p)
    text = f"{field} {len(sums)}\n" + "".join(
        f"{len(c)}\n" + "".join(f"{a:064x} {b:064x}\n" for a, b in c) for c in sums)
    out = subprocess.run([checker], input=text, capture_output=True, text=True, check=True, timeout=120).stdout
    inv = pow(R, -1, p)
    for c, line in zip(sums, out.splitlines(), strict=True):
        assert int(line, 16) == sum(a * b for a, b in c) * inv % p, c
