"""The device's Montgomery product, square and reduction against integers, at
the values where a carry chain can go wrong: limbs of all ones, single limbs,
values next to the modulus, zero, and random ones."""
import os
import random
import subprocess

import pytest

import apogee_gpu as A

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "field_check")
    import build_lib

    subprocess.check_call([build_lib._nvcc()] + build_lib.ARCH +
                          ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-o", exe,
                           os.path.join(HERE, "native", "field_check.cu")])
    return exe


def edge_values(p, rng):
    ones = (1 << 32) - 1
    vals = [0, 1, 2, p - 1, p - 2, p // 2, (1 << 256) % p, pow(1 << 256, -1, p)]
    vals += [1 << (32 * k) for k in range(8)] + [ones << (32 * k) for k in range(7)]
    vals += [(1 << (32 * k)) - 1 for k in range(1, 8)] + [p - (1 << (32 * k)) for k in range(8)]
    vals += [sum(ones << (32 * k) for k in range(s, 7, 2)) for s in (0, 1)]
    vals += [p - 1 - rng.randrange(1 << 40) for _ in range(8)] + [rng.randrange(p) for _ in range(32)]
    return [v % p for v in vals]


@pytest.mark.parametrize("field,p", [("q", A.P_Q), ("r", A.P_R)])
def test_products_squares_reductions(checker, field, p):
    vals = edge_values(p, random.Random(7))
    pairs = [(a, b) for a in vals for b in vals]
    text = f"{field} {len(pairs)}\n" + "".join(f"{a:064x} {b:064x}\n" for a, b in pairs)
    out = subprocess.run([checker], input=text, capture_output=True, text=True, check=True, timeout=120).stdout
    inv = pow(1 << 256, -1, p)
    for (a, b), line in zip(pairs, out.splitlines(), strict=True):
        assert [int(x, 16) for x in line.split()] == [a * b * inv % p, a * a * inv % p, a * inv % p], (a, b)
