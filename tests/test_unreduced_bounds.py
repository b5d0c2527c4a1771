"""Largest values inside the doubling chain (xyzz_dbl_chain_oct) and the eight-lane
addition (xyzz_add_oct_pt) of crypto_b200/csrc/curve.cuh, whose sums between products
are not reduced: every first operand is below 2^(32N) - p, every word fits, and one
conditional subtraction makes each result canonical where the code takes it as such."""
import pytest

P_BLS = int(
    "1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f6241eabfffeb153ffffb9feffffffffaaab",
    16)
P_BN = int("30644e72e131a029b85045b68181585d97816a916871ca8d3c208c16d87cfd47", 16)


@pytest.fixture(params=[(P_BLS, 12), (P_BN, 8)], ids=["bls12_381", "bn254"])
def field(request):
    p, n = request.param
    R = 1 << (32 * n)

    def mul(a, b):  # the largest result: p + a b / R before its one subtraction
        assert a < R - p and b < R and p + a * b // R < R
        return max(p - 1, a * b // R)

    def once(v):  # reduce_once of a value of N words
        assert v < R
        return max(p - 1, v - p)

    return p, R, n == 12, mul, once


def test_chain(field):
    p, R, wide, mul, once = field
    X = Y = ZZ = ZZZ = X2 = C = D = p - 1
    for _ in range(3):  # bounds only: the second round is a fixed point
        n = p  # p - D
        t = C + n
        if not wide:
            t = once(t)
            assert t == p - 1
        u = 3 * C + 4 * n if wide else 3 * t + n
        assert max(t, u, 2 * D) < R
        Xn, U2, CU, T, YD, ZZ = mul(X, u), mul(u, u), mul(C, u), mul(D, t), mul(Y, D), mul(ZZ, 2 * D)
        assert max(Xn, CU, T, YD, ZZ) == p - 1
        yn = once(2 * T + p)  # 2 D t - C u + p
        if not wide:
            yn = once(yn)
            assert yn == p - 1
        X2, C, D, ZZZ = mul(X2, U2), mul(CU, U2), mul(yn, 2 * yn), mul(ZZZ, 4 * YD)
        assert max(X2, C, D, ZZZ) == p - 1 and 4 * YD < R
        X, Y = Xn, yn
    assert once(Y) == p - 1


def test_eight_lane_addition(field):
    p, R, _, mul, _ = field
    c = mul(p - 1, p - 1)
    assert c == p - 1
    assert mul(c, 3 * c + c) == p - 1  # PP (3 R U1 + E P)
