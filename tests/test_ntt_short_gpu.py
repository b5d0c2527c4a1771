"""Short Fr transforms on both sides of the line between a thread per element (up
to 148 blocks) and a thread per butterfly, against the oracle."""
import pytest

import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("log_n", [1, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("batch", [1, 148, 149])
def test_short_vectors(cuda_lib, curve, log_n, batch):
    import torch

    import crypto_b200 as kb
    n = 1 << log_n
    data = kb.gen_scalars(curve, 7 * log_n + batch, n * batch)
    for inverse, coset in ((0, 0), (1, 1)):
        d = torch.frombuffer(bytearray(data), dtype=torch.uint8).cuda()
        assert kb.lib().kb200_ntt_device(curve, d.data_ptr(), n, inverse, coset, batch, None) == 0
        torch.cuda.synchronize()
        got = bytes(d.cpu().numpy().tobytes())
        for v in sorted({0, batch // 2, batch - 1}):
            part = slice(32 * n * v, 32 * n * (v + 1))
            assert got[part] == O.ntt(curve, data[part], inverse=bool(inverse), coset=bool(coset)), v
