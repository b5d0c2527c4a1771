"""G1 membership of EIP-2537 entries on both sides of the line between the
eight-lane and the one-thread test: a point outside G1 sets the status and
counts as infinity, wherever it stands."""
import random

import pytest

import _eip2537 as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 7168, 7169])
def test_points_outside_g1(cuda_lib, n):
    import torch

    import crypto_b200 as kb
    rng = random.Random(n)
    sc = kb.gen_scalars(2, n, n)
    d_ks = torch.frombuffer(bytearray(kb.gen_scalars(2, n + 1, n)), dtype=torch.uint8).cuda()
    d_pts = torch.empty(n * 96, dtype=torch.uint8, device="cuda")
    assert kb.lib().kb200_g1_fixed_base_device(2, d_ks.data_ptr(), n, d_pts.data_ptr(), None) == 0
    torch.cuda.synchronize()
    pts = bytes(d_pts.cpu().numpy().tobytes())
    ents = [E.entry(pts[96 * i:96 * i + 96], int.from_bytes(sc[32 * i:32 * i + 32], "little"))
            for i in range(n)]
    two = (0).to_bytes(48, "big") + (2).to_bytes(48, "big")  # order 3
    bad = {n - 1: E.curve_point_not_in_g1(rng), 0: E.torsion_point(rng), n // 2: two}
    for drop in ({}, bad):
        e, p, s = list(ents), [], []
        for i in range(n):
            if i in drop:
                e[i] = E.entry(drop[i], 7)
            else:
                p.append(pts[96 * i:96 * i + 96])
                s.append(sc[32 * i:32 * i + 32])
        d_in = torch.frombuffer(bytearray(b"".join(e)), dtype=torch.uint8).cuda()
        d_out = torch.ones(96, dtype=torch.uint8, device="cuda")
        d_st = torch.full((1,), 9, dtype=torch.int32, device="cuda")
        assert kb.lib().kb200_bls12_381_g1_msm_device(d_in.data_ptr(), 160 * n, d_out.data_ptr(),
                                                      d_st.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert int(d_st.item()) == (1 if drop else 0)
        want = kb.gpukit_multi_pippenger(2, b"".join(s), b"".join(p), len(p))
        assert bytes(d_out.cpu().numpy().tobytes()) == want
