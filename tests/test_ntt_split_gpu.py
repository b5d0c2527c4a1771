"""Fr transforms on both sides of the pass rules: single-block, cluster and
multi-pass sizes, batches around the lines between them."""
import pytest

import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("log_n,batch,inverse,coset", [
    (9, 3, 0, 1), (10, 1, 0, 1), (10, 148, 1, 0), (10, 149, 1, 0), (11, 2, 1, 1), (12, 1, 0, 0),
    (12, 5, 1, 1), (13, 1, 0, 1), (13, 40, 1, 0), (14, 3, 1, 1), (15, 1, 0, 0), (16, 1, 1, 1), (17, 1, 0, 0),
])
def test_batched_device_transform(cuda_lib, curve, log_n, batch, inverse, coset):
    import torch

    import crypto_b200 as kb
    n = 1 << log_n
    data = kb.gen_scalars(curve, 31 * log_n + batch, n * batch)
    d = torch.frombuffer(bytearray(data), dtype=torch.uint8).cuda()
    assert kb.lib().kb200_ntt_device(curve, d.data_ptr(), n, inverse, coset, batch, None) == 0
    torch.cuda.synchronize()
    got = bytes(d.cpu().numpy().tobytes())
    for v in sorted({0, 1, batch // 2, batch - 1}):
        if v < batch:
            part = slice(32 * n * v, 32 * n * (v + 1))
            assert got[part] == O.ntt(curve, data[part], inverse=bool(inverse), coset=bool(coset)), v


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("log_n", [9, 10, 12, 13, 16])
def test_noalloc_same_passes(cuda_lib, curve, log_n):
    import crypto_b200 as kb
    data = kb.gen_scalars(curve, log_n, 1 << log_n)
    for inverse in (False, True):
        for coset in (False, True):
            assert kb.ntt_fr_noalloc(curve, data, inverse, coset) == kb.ntt_fr(curve, data, inverse, coset)
