"""Word-prime transforms with even moduli, whose stages run one at a time in small
tiles and in pairs in full ones, from host-made stage tables: every one-line size,
two-pass and six-step sizes, against the oracle on unreduced 64-bit inputs."""
import numpy as np
import pytest

import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn", list(range(1, 15)) + [16, 17, 19])
@pytest.mark.parametrize("q,root", [(2, 1), ((1 << 40) + 6, 3), ((1 << 64) - 2, (1 << 63) + 5)])
def test_even_modulus(cuda_lib, logn, q, root):
    import crypto_b200 as kb
    x = np.random.Generator(np.random.PCG64(logn)).bit_generator.random_raw(1 << logn).astype(np.uint64)
    for inv in (False, True):
        got = x.copy()
        rc = kb.word_ntt_rc(got, len(got), q, root, inv)
        orc_rc, want = O.word_ntt(x, q, root, inv)
        assert rc == orc_rc == 0
        assert np.array_equal(got, want), inv
