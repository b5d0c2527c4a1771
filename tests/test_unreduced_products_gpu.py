"""The two-accumulator product beyond canonical operands: second operands of any
N words, operands whose even or odd words are all ones, and (inside the check)
multiples of p added to both operands."""
import ctypes
import random

import pytest

import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [0, 1, 2, 3])
def test_unreduced_operands(cuda_lib, field):
    import crypto_b200 as kb
    p = {0: O.FP[2], 1: O.FR[2], 2: O.FP[1], 3: O.FR[1]}[field]
    nb = 48 if field == 0 else 32
    full = 1 << (8 * nb)
    ones = sum(0xFFFFFFFF << (64 * i) for i in range(nb // 8))  # even words
    rng = random.Random(field)
    # Montgomery forms 0, 1, p - 1 and all-ones words at even and odd places, and
    # wide values, which the conversion multiplies as they are
    forms = [0, 1, p - 1, p - 2, ones % p, (ones << 32) % full % p, ones & (p >> 33), (ones << 32) & (p >> 1)]
    vals = [f * pow(full, -1, p) % p for f in forms]
    vals += [full - 1, full - p, ones, (ones << 32) % full, p, p + 1, full // p * p]
    vals += [rng.randrange(full) for _ in range(49)]
    A = [a for a in vals for _ in vals]
    B = vals * len(vals)
    le = lambda v: b"".join(x.to_bytes(nb, "little") for x in v)
    om, osq = (ctypes.create_string_buffer(len(A) * nb) for _ in range(2))
    bad = ctypes.c_ulonglong(1)
    assert kb.lib().kb200_field_mul_check(field, le(A), le(B), len(A), om, osq, ctypes.byref(bad)) == 0
    assert bad.value == 0
    assert om.raw == le([a * b % p for a, b in zip(A, B)])
    assert osq.raw == le([a * a % p for a in A])
