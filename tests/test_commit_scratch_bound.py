"""The commit server's admission bound per request against what a batch sets aside
for it, computed from the layout: entries, buckets, reduction results, evaluations.
A short polynomial joins a batch's 13-bit group, and a tuned class takes 16 or 19."""
import ctypes

import pytest


def use(n, c):
    """Bytes for one commit over shifted tables of c-bit windows, without pairing."""
    entries, buckets, point = (257 + c - 1) // c * n, 1 << (c - 1), 192
    blocks = min(128, -(-buckets // 256))  # of at most 256 buckets, 128 a window
    return (64 * n + 48 + 96 + 16 * entries + 12 * buckets + point * buckets
            + blocks * (16 * point + 4) + point)


@pytest.mark.parametrize("tuned", [0, 13, 16, 19])
def test_item_bound_covers_the_groups_a_commit_can_join(tuned):
    import crypto_b200 as kb
    bound = kb.lib()["_ZN5kb20025commit_item_scratch_bytesEm"]  # kb200::commit_item_scratch_bytes
    bound.restype, bound.argtypes = ctypes.c_size_t, [ctypes.c_size_t]
    for lg in range(21):
        kb.lib().kb200_tune_set(3, 2, lg, tuned)
        try:
            assert bound(1 << lg) >= use(1 << lg, tuned or 13), lg
        finally:
            kb.lib().kb200_tune_set(3, 2, lg, 0)
