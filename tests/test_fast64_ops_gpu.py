"""The branch-free quotients, roots and thirds of the FP64 kernels (csrc/fast64.cuh:
quo, inv64, sqrt64, third64) against the IEEE operators, over the operand ranges
their callers' tests accept: every exponent, mantissas next to powers of two,
signed zeros, and operands built to lie next to a rounding boundary."""
import pytest

from cumc3d_b200 import engine

pytestmark = pytest.mark.gpu

QUOTIENT, NEGATIVE, ROOT, THIRD, HARD, HARD_ANY, HARD_ROOT = range(7)


@pytest.mark.parametrize("what", [QUOTIENT, NEGATIVE, ROOT, THIRD])
def test_equal_the_ieee_operators(what):
    for seed in (1, 2, 3, 4):
        bad, ex = engine.check_fast64(what, seed * 0x9E3779B9, 1 << 28)
        assert bad == 0, (what, bad, ex)


def test_quotients_next_to_a_rounding_boundary():
    bad, ex = engine.check_fast64(HARD, 12345, 1 << 28)
    assert bad == 0, (bad, ex)
    # a divisor with a mantissa above 1.99 can round the other way, of such pairs
    # fewer than one in four million (their own chance is about 2^-52)
    bad, ex = engine.check_fast64(HARD_ANY, 12346, 1 << 28)
    assert bad < 1 << 6, (bad, ex)


def test_roots_next_to_a_rounding_boundary():
    bad, ex = engine.check_fast64(HARD_ROOT, 0, 8 * 400001)
    assert bad == 0, (bad, ex)


def test_unknown_kind_is_refused():
    with pytest.raises(engine.CumcError):
        engine.check_fast64(7, 1, 1)
