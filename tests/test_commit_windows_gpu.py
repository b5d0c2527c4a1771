"""KZG commits whose window size follows the polynomial's length (10 bits for up
to 256 evaluations, 13 above), alone and mixed in a batch, and the number of
bucket counts up to which one block scans: each commit against p(tau) G."""
import random

import pytest

import _oracle as O

pytestmark = pytest.mark.gpu

R = O.FR[2]
TAU = 0x1234567890ABCDEF1234567890ABCDEF1234567
SIZES = [1, 2, 64, 256, 512, 4096]


@pytest.fixture(scope="module")
def commits(cuda_lib):
    import crypto_b200 as kb
    kb.kzg_srs_generate(TAU.to_bytes(32, "little"), 4096)
    rng = random.Random(17)
    polys = {}
    for n in SIZES:
        coeffs = [rng.randrange(R) for _ in range(n)]
        y = 0
        for c in reversed(coeffs):
            y = (y * TAU + c) % R
        le = b"".join(c.to_bytes(32, "little") for c in coeffs)
        polys[n] = (O.ntt(2, le) if n > 1 else le, O.compress(O.g1_mul_gen(2, y)))
    return kb, polys


@pytest.mark.parametrize("n", SIZES)
def test_single(commits, n):
    kb, polys = commits
    assert kb.kzg_commit(polys[n][0]) == polys[n][1]


@pytest.mark.parametrize("sizes", [[2, 256, 64], [256] * 16, [64] * 17, [64, 512, 256], [1, 4096, 256, 512],
                                   [4096, 4096], [4096, 512, 2]])
def test_batch(commits, sizes):
    """Short ones alone (16 and 17 windows of 512: the last count one block scans
    and the first past it), short ones in the 13-bit group, two windows of 4096
    and three (likewise)."""
    kb, polys = commits
    got = kb.kzg_commit_batch(b"".join(polys[n][0] for n in sizes), sizes)
    assert list(got) == [polys[n][1] for n in sizes]
