"""The interpreter's round kernels: sumchecks of gate lists that they and no other
kernel run (interpreter_lists.py; test_round_kernel_choice.py holds which), round
by round against the oracle's restatement of gkr::prove_sumcheck
(crates/gkr/src/lib.rs:792)."""
import pytest

from interpreter_lists import LISTS, circuit
from test_gpu_gkr_sumcheck import check_circuit

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import apogee_gpu as A

    with A.Context(0) as c:
        yield c


@pytest.mark.parametrize("name", list(LISTS))
def test_rounds_match_oracle(ctx, name):
    check_circuit(ctx, circuit(name), 21, (0,))
